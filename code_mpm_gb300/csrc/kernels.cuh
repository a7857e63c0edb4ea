// Step kernels of the GB300 MPM engine.  One step of the reference's
// double-pass loop (PhysicsEngine_runSimulation_Classic_DoublePass_MPLocks.cpp:462-792,
// contact variant PhysicsEngine_runSimulation_Classic_DoublePass_MPLocks_Contact.cpp:27-543)
// maps onto:
//   k_reset_grid        ResetGrid (:4-22)
//   k_cell_keys         FindAGPs cell lookup, floor(x/h) (GridPoint_Mediator.cpp:8)
//   radix sort          particles ordered by cell key (on reorders, and where a step needs sorted cells)
//   k_cell_ranges       per-cell particle ranges (FP64 form, steps that detect contact)
//   k_p2g_cells         M2G (:48-89): each cell run's moments, then one atomic per corner and field;
//                       active-node marking (b_Active, :36)
//   k_step_lists        active-node list; DisplacementControl's claims (:143-174, last writer in
//                       list order); the device clock of a replayed step (engine.cu)
//   k_node_phase_a      displacement control, IntegrateGrid (:90-142; contact :242-277),
//                       f/m per node (the divisor of G2P pass 1)
//   k_pass1_remap       G2P pass 1 (:489-510) fused with the velocity remap (:539-564)
//   k_node_phase_b      v_i += (sum N m_p v_p) / m_i, displacement control, BC reapply
//                       (:573-599), p/m and v per node
//   k_pass2             G2P_P2_SmallStrain (:175-280; contact :438-525) fused with the
//                       constitutive increment and the platen timeline (:766-789)
//   k_contact_*         contact detection (…_Contact.cpp:152-237), bit-exact
#pragma once

#include "common.cuh"
#include "physics.cuh"
#include "surrogate.cuh"

namespace mpm {

// ---------------------------------------------------------------------------
// grid reset: zero every node that was active (the reference only clears
// active nodes; inactive ones are already zero).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_reset_grid(NView<T> nd, int contact) {
    step_enter<sizeof(T) == 4>();
    const long long nn = nd.nn;
    NODE_LOOP(nd, i) {
        unsigned st = nd.state[i];
        if (!(st & 1u)) continue;
        nd.state[i] = contact ? 0u : (st & ~(1u | NODE_CLAIMED));
        const Quad<T> z{(T)0, (T)0, (T)0, (T)0};
        *reinterpret_cast<Quad<T>*>(nd.acc + 8 * i) = z;
        *reinterpret_cast<Quad<T>*>(nd.acc + 8 * i + 4) = z;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (contact) nd.mg[c * nn + i] = 0.0;
            nd.vel[c * nn + i] = (T)0;
            nd.ftemp[c * nn + i] = (T)0;
        }
    }
}

// ---------------------------------------------------------------------------
// cell keys: base cell b = floor(x/h) per axis with the correctly rounded
// quotient, as glm::floor(d3Position / d3_Length_Cell)
// (GridPoint_Mediator.cpp:8), so the cell index is bit-identical to the
// reference.  Particles whose base cell lies outside [-1, cells] have no node
// in range and get key_max.  Decided in float-float arithmetic (fps_cell)
// unless the quotient lies within 1e-4 of an integer, then by the exact FP64
// quotient (cell_and_local).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned particle_key(const Geom& g, const double x[3], float u[3], unsigned* err) {
    bool ok = true;
    int b[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float ff;
        if (fps_cell(x[a], g.inv_hf[a], g.ih_lo[a], &ff, &u[a])) {
            if (ff < -1.0f || ff > (float)(g.nn[a] - 1)) ok = false;
            b[a] = ok ? (int)ff : 0;
            continue;
        }
        double f;
        if (!cell_and_local(g, a, x[a], f, u[a])) {
            atomicOr(err, ERR_NONFINITE_POSITION);
            ok = false;
            b[a] = 0;
            continue;
        }
        if (f < -1.0 || f > (double)(g.nn[a] - 1)) ok = false;
        b[a] = ok ? (int)f : 0;
    }
    return ok ? g.key_off + (unsigned)((b[0] + 1) + g.kd[0] * ((b[1] + 1) + g.kd[1] * (b[2] + 1))) : g.key_max;
}

static __global__ void k_cell_keys(const double* pos, long long n, Geom g, unsigned* keys, unsigned* vals,
                                   unsigned* keys_copy, unsigned* err, float* loc, const uint16_t* __restrict__ sid) {
    step_enter<true>();
    long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const double x[3] = {pos[p], pos[n + p], pos[2 * n + p]};
    float u[3];
    const unsigned key = particle_key(spec_geom(g, sid, p), x, u, err);
    keys[p] = key;
    if (keys_copy != keys) keys_copy[p] = key;
    if (vals) vals[p] = (unsigned)p;
    if (loc) {
#pragma unroll
        for (int a = 0; a < 3; ++a) loc[a * n + p] = u[a];
    }
}

// ---------------------------------------------------------------------------
// Per-cell [start, end) ranges in sorted order (for the FP64 form's exact
// contact gather, on output steps).
// ---------------------------------------------------------------------------
static __global__ void k_cell_ranges(const unsigned* __restrict__ skeys, long long n, Geom g,
                                     unsigned* __restrict__ cstart, unsigned* __restrict__ cend) {
    long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    unsigned key = skeys[s];
    if (key >= g.key_max) return;
    if (s == 0 || skeys[s - 1] != key) cstart[key] = (unsigned)s;
    if (s == n - 1 || skeys[s + 1] != key) cend[key] = (unsigned)(s + 1);
}

// ---------------------------------------------------------------------------
// Warp-segmented inclusive sum over runs of equal keys (sorted order puts a
// cell's particles in adjacent lanes); the run's last lane ends with the total.
// ---------------------------------------------------------------------------
struct Runs {
    int lane, head_lane, maxrun;
    bool tail;
    __device__ __forceinline__ void init(unsigned key) {
        lane = threadIdx.x & 31;
        unsigned kp = __shfl_up_sync(FULL_MASK, key, 1);
        unsigned kn = __shfl_down_sync(FULL_MASK, key, 1);
        bool head = (lane == 0) || (kp != key);
        tail = (lane == 31) || (kn != key);
        unsigned hm = __ballot_sync(FULL_MASK, head);
        head_lane = 31 - __clz(hm & (0xffffffffu >> (31 - lane)));
        maxrun = __reduce_max_sync(FULL_MASK, (unsigned)(lane - head_lane + 1));
    }
    template <typename T>
    __device__ __forceinline__ T sum(T v) const {
        for (int off = 1; off < maxrun; off <<= 1) {
            T o = __shfl_up_sync(FULL_MASK, v, off);
            if (lane - off >= head_lane) v += o;
        }
        return v;
    }
};

// Bases of particle p: FP64 form from the position, FP32 form from the
// cell-local coordinate the previous step stored (no FP64 instructions).
template <typename T>
__device__ __forceinline__ void load_place(const PView<T>& P, long long p, T x[3]) {
    const T* at;
    if constexpr (sizeof(T) == 4)
        at = P.loc;
    else
        at = P.pos;
#pragma unroll
    for (int c = 0; c < 3; ++c) x[c] = at[c * P.n + p];
}
template <typename T>
__device__ __forceinline__ void place_bases(const Geom& g, const T x[3], const int b[3], Bases<T>& B) {
    if constexpr (sizeof(T) == 4)
        B.init_local(g, x);
    else
        B.init(g, x, b);
}
template <typename T>
__device__ __forceinline__ void particle_bases(const PView<T>& P, const Geom& g, long long p, const int b[3],
                                               Bases<T>& B) {
    T x[3];
    load_place(P, p, x);
    place_bases(g, x, b, B);
}

// Prefetch into L2 the bytes of elements [p0, p0 + cnt) of an array of n
// ES-byte elements (a bulk prefetch, trimmed to 16-byte boundaries inside
// the array; a hint with no effect on results).
__device__ __forceinline__ void prefetch_l2(const void* base, int es, long long n, long long p0, int cnt) {
    if (!base) return;
    const unsigned long long lo = (unsigned long long)base, hi = lo + (unsigned long long)n * es;
    unsigned long long a = lo + (unsigned long long)p0 * es;
    unsigned long long b = lo + (unsigned long long)min((long long)n, p0 + cnt) * es;
    a = max(a & ~15ULL, (lo + 15) & ~15ULL);
    b = min((b + 15) & ~15ULL, hi & ~15ULL);
    if (b > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(b - a)) : "memory");
}

// ---------------------------------------------------------------------------
// P2G (M2G, …MPLocks.cpp:48-89): per particle and corner, mass N m, momentum
// N (m v), force -V (grad N . sigma) + N f_ext (Voigt order xx yy zz xy yz zx,
// :79-84), and (with_mg) the mass gradient grad N m of the contact path
// (…_Contact.cpp:131).  One thread per sorted slot.
//   REDUCE = 1: a cell's particles sit in adjacent lanes; their contributions
//               are summed across the lanes of the run first, then one atomic
//               per (node, field) per run.
//   REDUCE = 0: one atomic per (particle, node, field); the adds happen in L2.
// The choice (and the block size) is made per form by the autotuner.
// ---------------------------------------------------------------------------
template <typename T, int REDUCE>
__global__ void __launch_bounds__(512) k_p2g(PView<T> P, NView<T> nd, Geom g, const unsigned* skeys,
                                             const unsigned* perm, long long n, int with_mg) {
    step_enter<sizeof(T) == 4>();
    if (blockIdx.x == 0 && threadIdx.x == 0) *nd.acount = 0u;
    long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    unsigned key = (s < n) ? skeys[s] : 0xffffffffu;
    const bool valid = key < g.key_max;
    Runs run;
    if (REDUCE) run.init(key);
    else if (!valid) return;
    const long long np = P.n, nn = nd.nn;
    int b[3] = {0, 0, 0};
    Bases<T> B;
    T m = 0, vs[6] = {0, 0, 0, 0, 0, 0}, mv[3] = {0, 0, 0}, fe[3] = {0, 0, 0};
    const Geom* gsp = &g;
    if (valid) {
        long long p = perm[s];
        gsp = &spec_geom(g, P.sid, p);
        key_to_base(key, *gsp, b);
        particle_bases<T>(P, *gsp, p, b, B);
        m = P.mass[p];
        const T V = P.vol[p];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            mv[c] = m * P.vel[c * np + p];
            fe[c] = P.fext[c * np + p];
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) vs[c] = -V * P.stress[c * np + p];  // -V sigma
    }
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        T N = 0, G[3] = {0, 0, 0};
        if (valid) B.corner(k, N, G);
        T c[10];
        c[0] = N * m;
        c[1] = N * mv[0];
        c[2] = N * mv[1];
        c[3] = N * mv[2];
        c[4] = G[0] * vs[0] + G[1] * vs[3] + G[2] * vs[5] + N * fe[0];
        c[5] = G[1] * vs[1] + G[0] * vs[3] + G[2] * vs[4] + N * fe[1];
        c[6] = G[2] * vs[2] + G[0] * vs[5] + G[1] * vs[4] + N * fe[2];
        c[7] = G[0] * m;
        c[8] = G[1] * m;
        c[9] = G[2] * m;
        const int nf = with_mg ? 10 : 7;
        if (REDUCE) {
#pragma unroll
            for (int f = 0; f < 7; ++f) c[f] = run.sum(c[f]);
            if (with_mg) {
#pragma unroll
                for (int f = 7; f < 10; ++f) c[f] = run.sum(c[f]);
            }
        }
        if (valid && (!REDUCE || run.tail)) {
            long long nid = corner_node(*gsp, b, k);
            if (nid >= 0) {
                mark_active(nd.amark, (unsigned)nid);
                acc_add<T>(nd.acc, nid, c[0], c[1], c[2], c[3], c[4], c[5], c[6]);
                if (nf == 10) {
                    atomicAdd(&nd.mg[nid], c[7]);
                    atomicAdd(&nd.mg[nn + nid], c[8]);
                    atomicAdd(&nd.mg[2 * nn + nid], c[9]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// P2G, cell-centric (P2G modes 2 to 4).  A block takes BS consecutive slots.
// Phase 1: each slot's thread stages its particle's shape factors and transfer
// quantities in shared memory.  Phase 2: four threads per run of equal cell
// keys sum the run's contributions in slot order and issue one atomic per
// corner and field.
//
// What the four threads sum is the run's moments, not its corners.  With v =
// -V sigma and the trilinear N a corner's force is
//   -(sx FX(iy, iz) + sy FY(ix, iz) + sz FZ(ix, iy)) + sum N f_ext,
// s = +1/h at the lower and -1/h at the upper node of an axis, FX = sum over
// the particles of Ny Nz (v_xx, v_xy, v_xz) and FY, FZ likewise.  Thread (a, b)
// = (0..1, 0..1) keeps mass and momentum of the corners (ix, iy) = (a, b), iz =
// 0, 1, and the moments FX(a, b), FY(a, b), FZ(a, b): 22 multiply-adds per
// particle and thread against 39 when each thread formed its corners' forces,
// and the moments are exchanged by shuffles once per run.  This is what bounds
// the FP64 form (its FP64 pipe) and shortens the FP32 form's issue-bound sums.
//
// The gradient factors of a particle within 1e-12 of a node plane are zero
// (GridPoint_Mediator.cpp:118-133).  Its quantities are then staged as zero for
// that axis.  Where rounding leaves one of the axis' two factors (FP32: a
// cell-local coordinate below 3e-8), the staging thread adds that factor's
// share to the nodes itself (one particle in some ten million per step: every
// other step among 5M).
// ---------------------------------------------------------------------------
// Runs of equal cell keys among a block's slots: run r covers slots
// run_start[r] .. run_start[r + 1] - 1.  The slots need not be sorted (a cell met
// twice is two runs) and slots whose key is out of range form runs of their own,
// which the callers skip.  In two halves around the callers' staging, so that
// the block waits twice in all: run_heads (before) marks the warp's run heads
// from the keys, whose neighbours come by shuffle, and counts them; run_starts
// (after a __syncthreads) numbers them and ends with a __syncthreads (four waits
// before: P2G 135 -> 131 us on the 5.08M-particle batch, 33.1 -> 31.6 on the 1.07M block).
__device__ __forceinline__ unsigned run_heads(unsigned key, const unsigned* skeys, long long s, long long n,
                                              int* wsum) {
    const int t = threadIdx.x, lane = t & 31;
    unsigned prev = __shfl_up_sync(FULL_MASK, key, 1);
    if (lane == 0 && t > 0 && s < n) prev = skeys[s - 1];
    const unsigned heads = __ballot_sync(FULL_MASK, s < n && (t == 0 || prev != key));
    if (lane == 0) wsum[t >> 5] = __popc(heads);
    return heads;
}
template <int BS>
__device__ __forceinline__ int run_starts(unsigned heads, int nslots, int* run_start, const int* wsum) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int before = 0, R = 0;
#pragma unroll
    for (int k = 0; k < BS / 32; ++k) {
        const int x = wsum[k];
        if (k < w) before += x;
        R += x;
    }
    if ((heads >> lane) & 1u) run_start[before + __popc(heads & ((1u << lane) - 1u))] = t;
    if (t == 0) run_start[R] = nslots;
    __syncthreads();
    return R;
}

// FP32 cell-run value rows: slot s is stored at row position s ^ ((s >> 3) & 7),
// a permutation inside each aligned group of 8 slots (block sizes are multiples
// of 8).  The cell runs one warp sums start 8 slots apart when cells hold 8
// particles, so in slot order their 16-byte values fall in the same four banks
// and a quarter-warp's two runs conflict; swizzled, eight consecutive runs read
// eight distinct bank groups.  Sums still run in slot order.
__device__ __forceinline__ int slot_swz(int s) { return s ^ ((s >> 3) & 7); }

// The run arrays that follow the values: the slots' cell keys, the run starts
// (bs + 1) and the warps' run counts.
struct CellSlots {
    unsigned* key;
    int *run_start, *wsum;
    __device__ __forceinline__ CellSlots(unsigned char* at, int bs) {
        key = reinterpret_cast<unsigned*>(at);
        run_start = reinterpret_cast<int*>(key + bs);
        wsum = run_start + bs + 1;
    }
};
__host__ __device__ constexpr size_t cell_slots_bytes(int bs) { return (size_t)bs * 4 + (size_t)(bs + 1) * 4 + 64 * 4; }

// A slot's staged values, in rows of four (Quad): {m, m v}, {-V sigma xx xy zx,
// Nx0}, {xy yy yz, Ny0}, {zx yz zz, Nz0} (an axis' row zeroed when its gradient
// factors are), {f_ext, 0}; FP64: {Nx1, Ny1, Nz1, 0} (FP32: N1 = 1 - |u - 1| is
// 1 - N0 to the bit); FP32 with mass gradients: {m or 0 per axis, 0}.
// FP32: the axis rows carry the factor 1/h and the slot's corner nodes are
// staged too, so a run needs no geometry of its own; FP64: the 1/h and the
// nodes come once per run (nine FP64 products per particle less).
template <typename T>
__host__ __device__ constexpr int p2g_rows(bool mg) {
    return sizeof(T) == 8 || mg ? 6 : 5;
}
template <typename T>
__host__ __device__ constexpr size_t p2g_cells_smem(int bs, bool mg = false) {
    return (size_t)p2g_rows<T>(mg) * bs * 4 * sizeof(T) + (sizeof(T) == 4 ? bs * sizeof(CellNodes) : 0) +
           cell_slots_bytes(bs);
}

template <typename T>
__device__ __forceinline__ T quad_shfl(T v, int src) {
    return __shfl_sync(FULL_MASK, v, src);
}

template <typename T, int BS, bool FE, bool MG>
struct P2GBlock {
    using Q = Quad<T>;
    static constexpr bool F32 = sizeof(T) == 4;
    Q* row;
    CellNodes* nodes;  // FP32
    CellSlots cs;
    __device__ __forceinline__ explicit P2GBlock(unsigned char* raw)
        : row(reinterpret_cast<Q*>(raw)),
          nodes(reinterpret_cast<CellNodes*>(row + p2g_rows<T>(MG) * BS)),
          cs(reinterpret_cast<unsigned char*>(nodes + (F32 ? BS : 0)), BS) {
        static_assert(!MG || sizeof(T) == 4, "mass gradients: FP32 form");
    }

    // One gradient factor of an axis is zero and the other is not: the other's
    // share of the particle's force (and mass gradient), added to its four
    // nodes.  bit, step: the axis' corner bit and node stride; p, q: the other two
    // axes' shape factors, bits and strides.
    static __device__ __forceinline__ void lone_factor(const NView<T>& nd, const CellNodes& cn, int axis, int bit,
                                                       unsigned step, const T G[2], const T Np[2], int bitp,
                                                       unsigned stepp, const T Nq[2], int bitq, unsigned stepq, T v0,
                                                       T v1, T v2, T m) {
        const bool up = G[1] != (T)0;
        const T g = up ? G[1] : G[0];
        const unsigned n0 = cn.n0 + (up ? step : 0u);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int op = c >> 1, oq = c & 1;
            const int k = (up ? bit : 0) | (op ? bitp : 0) | (oq ? bitq : 0);
            if (!((cn.mask >> k) & 1u)) continue;
            const long long nid = n0 + (op ? stepp : 0u) + (oq ? stepq : 0u);
            const T w = -(Np[op] * Nq[oq]) * g;
            atomicAdd(nd.acc + 8 * nid + 4, w * v0);
            atomicAdd(nd.acc + 8 * nid + 5, w * v1);
            atomicAdd(nd.acc + 8 * nid + 6, w * v2);
            if constexpr (MG) atomicAdd(nd.mg + axis * nd.nn + nid, w * m);
        }
    }

    // slot t's particle: bases, mass m, volume V, velocity v, external force fe, stress sig
    __device__ __forceinline__ void stage(int t, const NView<T>& nd, const Geom& g, const int b[3], const Bases<T>& B,
                                          T m, T V, const T v[3], const T fe[3], const T sig[6]) const {
        static_assert(BS % 8 == 0, "slot swizzle groups");
        const int u = slot_swz(t);
        const bool x0 = B.gx[0] != (T)0, y0 = B.gy[0] != (T)0, z0 = B.gz[0] != (T)0;
        const bool x1 = B.gx[1] != (T)0, y1 = B.gy[1] != (T)0, z1 = B.gz[1] != (T)0;
        T s[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) s[c] = -V * sig[c];
        if (x0 != x1 || y0 != y1 || z0 != z1) {
            const CellNodes cn = cell_nodes(g, b);
            if (x0 != x1) lone_factor(nd, cn, 0, 4, 1u, B.gx, B.Ny, 2, cn.sy, B.Nz, 1, cn.sz, s[0], s[3], s[5], m);
            if (y0 != y1) lone_factor(nd, cn, 1, 2, cn.sy, B.gy, B.Nx, 4, 1u, B.Nz, 1, cn.sz, s[3], s[1], s[4], m);
            if (z0 != z1) lone_factor(nd, cn, 2, 1, cn.sz, B.gz, B.Nx, 4, 1u, B.Ny, 2, cn.sy, s[5], s[4], s[2], m);
        }
        const bool x = x0 && x1, y = y0 && y1, z = z0 && z1;
        const T o = (T)0;
        row[u] = Q{m, m * v[0], m * v[1], m * v[2]};
        if constexpr (F32) {
            const T hx = x ? B.gx[0] : o, hy = y ? B.gy[0] : o, hz = z ? B.gz[0] : o;
            row[BS + u] = Q{hx * s[0], hx * s[3], hx * s[5], B.Nx[0]};
            row[2 * BS + u] = Q{hy * s[3], hy * s[1], hy * s[4], B.Ny[0]};
            row[3 * BS + u] = Q{hz * s[5], hz * s[4], hz * s[2], B.Nz[0]};
            nodes[t] = cell_nodes(g, b);
        } else {
            row[BS + u] = Q{x ? s[0] : o, x ? s[3] : o, x ? s[5] : o, B.Nx[0]};
            row[2 * BS + u] = Q{y ? s[3] : o, y ? s[1] : o, y ? s[4] : o, B.Ny[0]};
            row[3 * BS + u] = Q{z ? s[5] : o, z ? s[4] : o, z ? s[2] : o, B.Nz[0]};
        }
        if constexpr (FE) row[4 * BS + u] = Q{fe[0], fe[1], fe[2], o};
        if constexpr (MG)
            row[5 * BS + u] = Q{x ? B.gx[0] * m : o, y ? B.gy[0] * m : o, z ? B.gz[0] * m : o, o};
        if constexpr (sizeof(T) == 8) row[5 * BS + u] = Q{B.Nx[1], B.Ny[1], B.Nz[1], o};
    }

    // After the staging and a __syncthreads (keys in cs.key for the first nslots
    // slots, out of range where nothing was staged; heads from run_heads): the runs' sums and their
    // atomics, which also mark the corners active.  MG: also the node
    // mass gradients.  sid: the slots' specimens from the block's first slot on
    // (perm: through the sort order), for the runs' geometry.
    //
    // FP32: a warp holds consecutive runs, the threads of a run in adjacent
    // lanes.  When run r's cell follows run r - 1's in x (key + 1), the x = 1
    // corners of r - 1 are the x = 0 corners of r: one shuffle of the sums, two
    // lanes up, adds them to r's, and only r's lanes issue the atomics (in the
    // honeycomb batch about three runs in four have such a neighbour, so a
    // third of the corner atomics go).
    __device__ __forceinline__ void scatter(const NView<T>& nd, const Geom& g, const uint16_t* __restrict__ sid,
                                            const unsigned* perm, long long s0, int nslots,
                                            unsigned heads) const {
        const int t = threadIdx.x, lane = t & 31;
        const long long nn = nd.nn;
        const unsigned* skey = cs.key;
        const int R = run_starts<BS>(heads, nslots, cs.run_start, cs.wsum);
        const int nitems = R * 4;
        const int quad = lane & ~3, a = (t >> 1) & 1, b = t & 1;
        // whole warps take the loop together (the shuffles)
        for (int item = t; item - lane < nitems; item += BS) {
            const bool live = item < nitems;
            const int r = live ? item >> 2 : 0;
            const int first = cs.run_start[r];
            const unsigned key = skey[first];
            // slots outside the grid (and lanes past the items) sum nothing
            const bool inb = live && key < g.key_max;
            const int e = inb ? cs.run_start[r + 1] : first;
            T c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};          // {m, m v} of the corners iz = 0, 1
            T fx[3] = {0, 0, 0}, fy[3] = {0, 0, 0}, fz[3] = {0, 0, 0};  // moments (a, b)
            T e0[3] = {0, 0, 0}, e1[3] = {0, 0, 0};                // N f_ext
            T mx = 0, my = 0, mz = 0;                              // mass moments (MG)
#pragma unroll 1
            for (int i = first; i < e; ++i) {
                const int u = slot_swz(i);
                const Q q = row[u], X = row[BS + u], Y = row[2 * BS + u], Z = row[3 * BS + u];
                T nx1, ny1, nz1;
                if constexpr (sizeof(T) == 8) {
                    const Q N = row[5 * BS + u];
                    nx1 = N.x, ny1 = N.y, nz1 = N.z;
                } else {
                    nx1 = (T)1 - X.w, ny1 = (T)1 - Y.w, nz1 = (T)1 - Z.w;
                }
                const T nx = a ? nx1 : X.w, nya = a ? ny1 : Y.w, nyb = b ? ny1 : Y.w;
                const T nz0 = Z.w, nzb = b ? nz1 : nz0;
                const T A = nx * nyb, w0 = A * nz0, w1 = A * nz1, wx = nya * nzb, wy = nx * nzb;
                c0[0] += w0 * q.x, c0[1] += w0 * q.y, c0[2] += w0 * q.z, c0[3] += w0 * q.w;
                c1[0] += w1 * q.x, c1[1] += w1 * q.y, c1[2] += w1 * q.z, c1[3] += w1 * q.w;
                fx[0] += wx * X.x, fx[1] += wx * X.y, fx[2] += wx * X.z;
                fy[0] += wy * Y.x, fy[1] += wy * Y.y, fy[2] += wy * Y.z;
                fz[0] += A * Z.x, fz[1] += A * Z.y, fz[2] += A * Z.z;
                if constexpr (FE) {
                    const Q f = row[4 * BS + u];
                    e0[0] += w0 * f.x, e0[1] += w0 * f.y, e0[2] += w0 * f.z;
                    e1[0] += w1 * f.x, e1[1] += w1 * f.y, e1[2] += w1 * f.z;
                }
                if constexpr (MG) {
                    const Q M = row[5 * BS + u];
                    mx += wx * M.x, my += wy * M.y, mz += A * M.z;
                }
            }
            // the run's geometry and corner nodes
            CellNodes cn{0u, 0u, 0u, 0u};
            T hx = 1, hy = 1, hz = 1;  // 1/h where the staged rows do not carry it
            if constexpr (F32) {
                if (inb) cn = nodes[first];
            } else if (inb) {
                const Geom& gs = (g.nspec > 1) ? g.tab[sid[perm ? perm[s0 + first] : s0 + first]] : g;
                int base[3];
                key_to_base(key, gs, base);
                cn = cell_nodes(gs, base);
                hx = gs.inv_h[0];
                hy = gs.inv_h[1];
                hz = gs.inv_h[2];
            }
            if (a == 0) hx = -hx;  // -s of this thread's corners (ix, iy) = (a, b)
            if (b == 0) hy = -hy;
            T p0[3], p1[3], g0[3], g1[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T X0 = quad_shfl(fx[c], quad + 2 * b), X1 = quad_shfl(fx[c], quad + 2 * b + 1);
                const T Y0 = quad_shfl(fy[c], quad + 2 * a), Y1 = quad_shfl(fy[c], quad + 2 * a + 1);
                p0[c] = hx * X0 + hy * Y0 - hz * fz[c];
                p1[c] = hx * X1 + hy * Y1 + hz * fz[c];
                if constexpr (FE) p0[c] += e0[c], p1[c] += e1[c];
            }
            if constexpr (MG) {
                g0[0] = hx * quad_shfl(mx, quad + 2 * b), g1[0] = hx * quad_shfl(mx, quad + 2 * b + 1);
                g0[1] = hy * quad_shfl(my, quad + 2 * a), g1[1] = hy * quad_shfl(my, quad + 2 * a + 1);
                g0[2] = -hz * mz, g1[2] = hz * mz;
            }
            bool skip = !inb;
            if constexpr (sizeof(T) == 4) {
                constexpr int SH = 2;  // lanes from run r - 1's x = 1 corners to run r's x = 0 corners
                const bool recv = inb && !a && lane >= SH && r > 0 && skey[cs.run_start[r - 1]] + 1u == key;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float x0 = __shfl_up_sync(FULL_MASK, c0[c], SH), x1 = __shfl_up_sync(FULL_MASK, c1[c], SH);
                    if (recv) c0[c] += x0, c1[c] += x1;
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float x0 = __shfl_up_sync(FULL_MASK, p0[c], SH), x1 = __shfl_up_sync(FULL_MASK, p1[c], SH);
                    if (recv) p0[c] += x0, p1[c] += x1;
                    if constexpr (MG) {
                        const float y0 = __shfl_up_sync(FULL_MASK, g0[c], SH);
                        const float y1 = __shfl_up_sync(FULL_MASK, g1[c], SH);
                        if (recv) g0[c] += y0, g1[c] += y1;
                    }
                }
                // a sender's sums went to the lane SH up (lanes near the warp's top read their own false)
                if (__shfl_down_sync(FULL_MASK, recv ? 1 : 0, SH) && a) skip = true;
            }
            if (skip) continue;
            const unsigned n0 = cn.n0 + a + (b ? cn.sy : 0u);
            const unsigned ok = cn.mask >> (4 * a + 2 * b);
#pragma unroll
            for (int iz = 0; iz < 2; ++iz) {
                if (!((ok >> iz) & 1u)) continue;
                const long long nid = iz ? n0 + cn.sz : n0;
                const T* c = iz ? c1 : c0;
                const T* f = iz ? p1 : p0;
                // active nodes: the in-range corners of occupied cells (b_Active, …MPLocks.cpp:36)
                mark_active(nd.amark, (unsigned)nid);
                acc_add<T>(nd.acc, nid, c[0], c[1], c[2], c[3], f[0], f[1], f[2]);
                if constexpr (MG) {
                    const T* gm = iz ? g1 : g0;
                    atomicAdd(&nd.mg[nid], gm[0]);
                    atomicAdd(&nd.mg[nn + nid], gm[1]);
                    atomicAdd(&nd.mg[2 * nn + nid], gm[2]);
                }
            }
        }
    }
};

// FE: some particle carries an external force (uploaded; without one the forces are not read).  MG: also the contact
// path's node mass gradients (output steps of the FP32 form).
template <typename T, int BS, bool FE, bool MG>
__device__ __forceinline__ void p2g_cells_run(const PView<T>& P, const NView<T>& nd, const Geom& g,
                                              const unsigned* skeys, const unsigned* perm,
                                              long long n) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const P2GBlock<T, BS, FE, MG> blk(smem_raw);
    step_enter<sizeof(T) == 4>();
    const int t = threadIdx.x;
    if (blockIdx.x == 0 && t == 0) *nd.acount = 0u;
    const long long s0 = blockIdx.x * (long long)BS, s = s0 + t;
    const unsigned key = (s < n) ? skeys[s] : 0xffffffffu;
    const unsigned heads = run_heads(key, skeys, s, n, blk.cs.wsum);
    const long long np = P.n;
    if (key < g.key_max) {
        const long long p = perm ? perm[s] : s;
        const Geom& gs = spec_geom(g, P.sid, p);
        int b[3];
        key_to_base(key, gs, b);
        Bases<T> B;
        particle_bases<T>(P, gs, p, b, B);
        T v[3], fe[3] = {0, 0, 0}, sig[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = P.vel[c * np + p];
        if constexpr (FE) {
#pragma unroll
            for (int c = 0; c < 3; ++c) fe[c] = P.fext[c * np + p];
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) sig[c] = P.stress[c * np + p];
        blk.stage(t, nd, gs, b, B, P.mass[p], P.vol[p], v, fe, sig);
    }
    blk.cs.key[t] = key;
    __syncthreads();
    blk.scatter(nd, g, P.sid, perm, s0, (int)min((long long)BS, n - s0), heads);
}

// Threads resident per SM that the FP32 kernels are built for (P2G: 1280 at 48
// registers; 5.08M particles of honeycombs, 138 us, against 140 us for 1536 at
// 40 registers with spills and 176 us for 1024).  Before the moments P2G took
// 154 us there (now 131), 39.1 us (now 31.6) on a solid block of 1.07M particles; FP64
// form, a solid block of 286k particles: 233 us before, 112 now.
template <typename T, int BS, bool FE>
__global__ void __launch_bounds__(BS, sizeof(T) == 4 ? 1280 / BS : 1) k_p2g_cells(
    PView<T> P, NView<T> nd, Geom g, const unsigned* skeys, const unsigned* perm, long long n) {
    p2g_cells_run<T, BS, FE, false>(P, nd, g, skeys, perm, n);
}

template <int BS>
__global__ void __launch_bounds__(BS) k_p2g_cells_mg(PView<float> P, NView<float> nd, Geom g,
                                                      const unsigned* skeys, const unsigned* perm, long long n) {
    p2g_cells_run<float, BS, true, true>(P, nd, g, skeys, perm, n);
}

// ---------------------------------------------------------------------------
// Displacement control (…MPLocks.cpp:143-174; contact :283-297, :416-432).
// The reference overwrites node velocity/momentum/force from each controlled
// particle in list order, so a node shared by several keeps the last one's.
// dc_claim records, per node and axis, the largest list position writing
// it, and marks the node (NODE_CLAIMED in its state word) so the node phases
// read the claims of marked nodes only; node_dc lets only the claiming
// particle write.  contact: every particle claims all three axes, so the axis-0
// claim word stands for the three (one atomic per corner instead of three).
// ---------------------------------------------------------------------------
// Called by whole warps, lane by lane along the list (k < ndc: this lane has an
// entry).  A claim is lost where the next entry claims the same nodes and axes,
// as neighbours in a platen's list mostly do, two to a cell: it is not made (the
// atomics of one cell queue: 24.4 -> 17.4 us on the 5.08M-particle batch).
__device__ __forceinline__ void dc_claim(int k, int ndc, const unsigned* __restrict__ dclist,
                                         const unsigned* keys, const uint8_t* pflags,
                                         const Geom& g, unsigned* owner, long long nn, int contact,
                                         const uint16_t* __restrict__ sid, unsigned* state) {
    const bool have = k < ndc;
    const unsigned p = have ? dclist[k] : 0u;
    const unsigned key = have ? keys[p] : 0xffffffffu;
    const unsigned axes = contact ? 7u : have ? pflags[p] & 7u : 0u;
    const unsigned next_key = __shfl_down_sync(FULL_MASK, key, 1), next_axes = __shfl_down_sync(FULL_MASK, axes, 1);
    if (!(key < g.key_max) || !axes) return;
    if ((threadIdx.x & 31) < 31 && next_key == key && next_axes == axes) return;
    const Geom& gs = spec_geom(g, sid, p);
    int b[3];
    key_to_base(key, gs, b);
    const CellNodes cn = cell_nodes(gs, b);
#pragma unroll
    for (int c8 = 0; c8 < 8; ++c8) {
        if (!((cn.mask >> c8) & 1u)) continue;
        const long long nid = cell_node(cn, c8);
        for (int a = 0; a < 3; ++a)
            if ((axes & (1u << a)) && !(contact && a > 0)) atomicMax(&owner[a * nn + nid], (unsigned)k + 1u);
        atomicOr(&state[nid], NODE_CLAIMED);
    }
}

// ---------------------------------------------------------------------------
// Grid momentum update with boundary conditions (IntegrateGrid,
// …MPLocks.cpp:90-142).  Non-contact order: damping, x-wall Coulomb friction
// on y (:106-124), zero fixed axes (y-fixed nodes accumulate the reaction
// force, :129), then p += f dt.  Contact order (…_Contact.cpp:250-276):
// damping, p += f dt, then zero fixed axes; optionally Coulomb friction on
// the x/y tangents of z-fixed nodes (floor_friction, an extension).
// Damping is skipped when its coefficient is zero (f - 0*x == f).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void coulomb(T p_t, T& f_t, T fn, T mu, T dt) {
    T trial = p_t + f_t * dt;
    T ff = mu * (T)((T(0) < -trial) - (-trial < T(0))) * fabs(fn);
    if (fabs(ff * dt) > fabs(trial)) ff *= fabs(trial / dt) / fabs(ff);
    f_t += ff;
}

// The update of one node's momentum p and force f in registers; zero[c]: the
// axis is fixed (its velocity is zeroed too); ft_y: the y reaction force of a
// y-fixed node.  friction is read only where a friction law applies.
template <typename T>
__device__ __forceinline__ void grid_update_regs(const NView<T>& nd, long long i, unsigned fx, T p[3], T f[3], T dt,
                                                 double damping, int contact, int floor_friction, bool zero[3],
                                                 T& ft_y, T dfr[3]) {
    dfr[0] = dfr[1] = dfr[2] = (T)0;  // the force each friction law added (for the friction work)
    if (damping != 0.0) {
        T pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
        if (sqrt(pp) > (T)1.0e-24) {
            T inv = (T)1 / sqrt(pp);
            T nrm[3] = {p[0] * inv, p[1] * inv, p[2] * inv};
            T sc = (T)damping * fabs(f[0] * nrm[0] + f[1] * nrm[1] + f[2] * nrm[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] = f[c] - sc * nrm[c];
        }
    }
    zero[0] = zero[1] = zero[2] = false;
    ft_y = 0;
    if (!contact) {
        if (fx & 1u) {
            T trial_y = p[1] + f[1] * dt;
            if (fabs(trial_y * dt) > (T)1.0e-24 && f[0] > (T)0) {
                const T f0 = f[1];
                coulomb<T>(p[1], f[1], f[0], (T)nd.friction[i], dt);
                dfr[1] = f[1] - f0;
            }
            zero[0] = true;
            p[0] = 0;
            f[0] = 0;
        }
        if (fx & 2u) {
            ft_y = f[1];
            zero[1] = true;
            p[1] = 0;
            f[1] = 0;
        }
        if (fx & 4u) {
            zero[2] = true;
            p[2] = 0;
            f[2] = 0;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) p[c] = p[c] + f[c] * dt;
    } else {
        if (floor_friction && (fx & 4u) && nd.friction[i] > 0.0 && f[2] < (T)0) {
            T fz = f[2], mu = (T)nd.friction[i];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                T trial = p[t] + f[t] * dt;
                if (fabs(trial * dt) > (T)1.0e-24) {
                    const T f0 = f[t];
                    coulomb<T>(p[t], f[t], fz, mu, dt);
                    dfr[t] = f[t] - f0;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) p[c] = p[c] + f[c] * dt;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (fx & (1u << c)) {
                if (c == 1) ft_y = f[1];
                zero[c] = true;
                p[c] = 0;
                f[c] = 0;
            }
        }
    }
}

// The factor dt of what the particles gather: the FP64 form takes it once per
// node, in the records (its FP64 operations bound it), the FP32 form in each
// particle, after the sum (pass2_particle says why).
__device__ __forceinline__ double record_dt(double x, double dt) { return x * dt; }
__device__ __forceinline__ float record_dt(float x, float) { return x; }
__device__ __forceinline__ double gather_dt(double x, double) { return x; }
__device__ __forceinline__ float gather_dt(float x, float dt) { return x * dt; }

// ---------------------------------------------------------------------------
// G2P pass 1 (…MPLocks.cpp:489-510): v_p += N (f_i/m_i) dt over the corners
// in findAdjacentGridPoints order, fused with the velocity remap (:539-564):
// each particle then scatters N m_p v_p, summed per run before the atomic.
// Contact path: particles flagged b_DisplacementControl are skipped.
// ---------------------------------------------------------------------------
template <typename T, int BATCH>
__global__ void __launch_bounds__(256) k_pass1_remap(PView<T> P, NView<T> nd, Geom g,
                                                     const unsigned* skeys, const unsigned* perm, long long n, T dt,
                                                     int contact) {
    step_enter<sizeof(T) == 4>();
    long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    unsigned key = (s < n) ? skeys[s] : 0xffffffffu;
    Runs run;
    run.init(key);
    // key_ok: the run has grid nodes (its tail lane issues the atomics even
    // when its own particle is skipped); valid: this particle takes part
    const bool key_ok = key < g.key_max;
    bool valid = key_ok;
    const long long np = P.n, nn = nd.nn;
    long long p = 0;
    const Geom* gsp = &g;
    int b[3] = {0, 0, 0};
    if (key_ok) {
        p = perm[s];
        if (contact && (P.pflags[p] & 8u)) valid = false;
        gsp = &spec_geom(g, P.sid, p);
        key_to_base(key, *gsp, b);
    }
    Bases<T> B;
    T m = 0, v[3] = {0, 0, 0};
    if (valid) {
        particle_bases<T>(P, *gsp, p, b, B);
        m = P.mass[p];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = P.vel[c * np + p];
        // BATCH: every corner's record is requested before any is used (one
        // round trip to memory instead of eight, at more registers); the sum
        // runs in corner order either way
        if constexpr (BATCH) {
            Quad<T> r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const long long nid = corner_node(*gsp, b, k);
                r[k] = nid >= 0 ? ld_quad(nd.rec + 8 * nid) : Quad<T>{(T)0, (T)0, (T)0, (T)0};
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (!(r[k].w != (T)0)) continue;  // out of range or m <= mass_min
                T N, G[3];
                B.corner(k, N, G);
                v[0] = v[0] + gather_dt(N * r[k].x, dt);
                v[1] = v[1] + gather_dt(N * r[k].y, dt);
                v[2] = v[2] + gather_dt(N * r[k].z, dt);
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < 8; ++k) {
                const long long nid = corner_node(*gsp, b, k);
                if (nid < 0) continue;
                const Quad<T> r = ld_quad(nd.rec + 8 * nid);
                if (!(r.w != (T)0)) continue;
                T N, G[3];
                B.corner(k, N, G);
                v[0] = v[0] + gather_dt(N * r.x, dt);
                v[1] = v[1] + gather_dt(N * r.y, dt);
                v[2] = v[2] + gather_dt(N * r.z, dt);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) P.vel[c * np + p] = v[c];
    }
    T mv[3] = {m * v[0], m * v[1], m * v[2]};
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        T N = 0, G[3];
        if (valid) B.corner(k, N, G);
        T q0 = run.sum(N * mv[0]);
        T q1 = run.sum(N * mv[1]);
        T q2 = run.sum(N * mv[2]);
        if (key_ok && run.tail) {
            long long nid = corner_node(*gsp, b, k);
            if (nid >= 0) {
                q_add<T>(nd.q, nid, q0, q1, q2);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// G2P pass 1 + velocity remap, cell-centric (used with P2G modes 2 to 4): each
// slot's thread updates its particle's velocity from the node records and
// stages N (per axis) and m v in shared memory; one thread per (cell run, CPT
// corners) then sums N m v over the run in slot order and issues one vector
// (FP64: three) atomics per corner.  Skipped particles (platen on the contact
// path) stay in their run with zero weight.
// Both forms work on the (x, y) pairs of corners: A = Nx Ny once, then N = A Nz
// (FP64: 96 operations per particle on the pipe that bounds it, from 190
// corner by corner with the records' thresholds tested; a record's r is zero
// where m <= mass_min).  A solid block of 286k particles in the FP64 form:
// 107 us before, 77 now.
// ---------------------------------------------------------------------------
// The slots' corner nodes, staged beside the keys: the first node, and the
// strides and mask of the cell.
template <typename T>
__host__ __device__ constexpr size_t pass1_cells_smem(int bs) {
    return (size_t)(sizeof(T) == 4 ? 9 : 10) * bs * sizeof(T) + (size_t)bs * sizeof(CellNodes) + cell_slots_bytes(bs);
}

// FP32 with 1 or 2 corners per thread: registers capped for 1536 resident
// threads per SM (40 registers), about 10% faster than 56 registers at 1152
// threads: the kernel waits on its record gathers, and more resident warps
// keep more of them in flight (1280 and 1024 threads with all eight records
// requested at once: 135 us against 118 on the 5.08M-particle batch).  A
// slot's particle fields are requested with its key rather than after it: 129
// -> 118 us there, 48.1 -> 44.7 on 1.89M particles, 26.9 -> 26.0 on 1.07M.
template <typename T, int CPT, int BS>
__global__ void __launch_bounds__(BS, sizeof(T) == 4 && CPT < 4 ? 1536 / BS : 1) k_pass1_cells(PView<T> P, NView<T> nd, Geom g,
                                                     const unsigned* skeys, const unsigned* perm, long long n, T dt,
                                                     int contact) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int bs = BS;
    const int t = threadIdx.x;
    // FP64: rows of bs pairs {Nx0 Nx1} {Ny0 Ny1} {Nz0 Nz1} {mv0 mv1} {mv2 0}.
    // FP32: two rows of bs float4 {Nx0 Nx1 Ny0 Ny1} {Nz0 Nz1 mv0 mv1} and a row of mv2.
    constexpr bool F32 = sizeof(T) == 4;
    static_assert(BS % 8 == 0, "slot swizzle groups");
    CellNodes* scn = reinterpret_cast<CellNodes*>(smem_raw);
    T* sn = reinterpret_cast<T*>(scn + bs);
    CellSlots cs(reinterpret_cast<unsigned char*>(sn + (F32 ? 9 : 10) * bs), bs);
    unsigned* skey = cs.key;
    step_enter<sizeof(T) == 4>();
    const long long s = blockIdx.x * (long long)bs + t;
    const long long np = P.n;
    const unsigned key = (s < n) ? skeys[s] : 0xffffffffu;
    const long long p = s < n ? (perm ? perm[s] : s) : 0;
    T x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, m = 0;
    bool valid = true;
    if (s < n) {
        load_place(P, p, x);
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = P.vel[c * np + p];
        m = P.mass[p];
        valid = !(contact && (P.pflags[p] & 8u));
    }
    const unsigned heads = run_heads(key, skeys, s, n, cs.wsum);
    if (key < g.key_max) {
        const Geom& gs = spec_geom(g, P.sid, p);
        int b[3];
        key_to_base(key, gs, b);
        const CellNodes cn = cell_nodes(gs, b);
        scn[t] = cn;
        T N6[6] = {0, 0, 0, 0, 0, 0}, mv[3] = {0, 0, 0};
        if (valid) {
            Bases<T> B;
            place_bases<T>(gs, x, b, B);
            // four corners' records requested before any is used; summed in corner order
#pragma unroll(F32 ? 2 : 1)
            for (int h = 0; h < 2; ++h) {
                Quad<T> rq[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = 4 * h + j;
                    const Quad<T> z{(T)0, (T)0, (T)0, (T)0};
                    rq[j] = ((cn.mask >> k) & 1u) ? ld_quad(nd.rec + 8ll * cell_node(cn, k)) : z;
                }
                const T nx = h ? B.Nx[1] : B.Nx[0];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const T N = nx * ((j & 2) ? B.Ny[1] : B.Ny[0]) * ((j & 1) ? B.Nz[1] : B.Nz[0]);
                    v[0] += gather_dt(N * rq[j].x, dt);
                    v[1] += gather_dt(N * rq[j].y, dt);
                    v[2] += gather_dt(N * rq[j].z, dt);
                }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                P.vel[c * np + p] = v[c];
                mv[c] = m * v[c];
            }
            N6[0] = B.Nx[0];
            N6[1] = B.Nx[1];
            N6[2] = B.Ny[0];
            N6[3] = B.Ny[1];
            N6[4] = B.Nz[0];
            N6[5] = B.Nz[1];
        }
        const int u = slot_swz(t);
        if constexpr (F32) {
            float4* sv = reinterpret_cast<float4*>(sn);
            sv[u] = make_float4(N6[0], N6[1], N6[2], N6[3]);
            sv[bs + u] = make_float4(N6[4], N6[5], mv[0], mv[1]);
            sn[8 * bs + u] = mv[2];
        } else {
            double2* sv = reinterpret_cast<double2*>(sn);
            sv[u] = make_double2(N6[0], N6[1]);
            sv[bs + u] = make_double2(N6[2], N6[3]);
            sv[2 * bs + u] = make_double2(N6[4], N6[5]);
            sv[3 * bs + u] = make_double2(mv[0], mv[1]);
            sv[4 * bs + u] = make_double2(mv[2], 0.0);
        }
    }
    skey[t] = key;
    __syncthreads();
    const int R = run_starts<BS>(heads, (int)min((long long)bs, n - blockIdx.x * (long long)bs), cs.run_start, cs.wsum);
    constexpr int TPR = 8 / CPT;  // threads per run; each sums CPT corners sharing its x (and y) bases
    for (int item = t; item < R * TPR; item += bs) {
        const int r = item / TPR, k0 = (item % TPR) * CPT;
        const int a = cs.run_start[r], e = cs.run_start[r + 1];
        if (!(skey[a] < g.key_max)) continue;  // slots outside the grid
        T q0[CPT], q1[CPT], q2[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) q0[j] = q1[j] = q2[j] = 0;
        for (int i = a; i < e; ++i) {
            const int u = slot_swz(i);
            T mv0, mv1, mv2, X[2], Y[2], Z[2];
            if constexpr (F32) {
                const float4* sv = reinterpret_cast<const float4*>(sn);
                const float4 A = sv[u], B = sv[bs + u];
                X[0] = A.x, X[1] = A.y, Y[0] = A.z, Y[1] = A.w, Z[0] = B.x, Z[1] = B.y;
                mv0 = B.z, mv1 = B.w, mv2 = sn[8 * bs + u];
            } else {
                const double2* sv = reinterpret_cast<const double2*>(sn);
                const double2 A = sv[u], B = sv[bs + u], C = sv[2 * bs + u], D = sv[3 * bs + u];
                X[0] = A.x, X[1] = A.y, Y[0] = B.x, Y[1] = B.y, Z[0] = C.x, Z[1] = C.y;
                mv0 = D.x, mv1 = D.y, mv2 = sv[4 * bs + u].x;
            }
            const T nx = (k0 & 4) ? X[1] : X[0];
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const int k = k0 + j;
                const T N = nx * ((k & 2) ? Y[1] : Y[0]) * ((k & 1) ? Z[1] : Z[0]);
                q0[j] += N * mv0;
                q1[j] += N * mv1;
                q2[j] += N * mv2;
            }
        }
        const CellNodes cn = scn[a];
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
            const int k = k0 + j;
            if ((cn.mask >> k) & 1u) q_add<T>(nd.q, cell_node(cn, k), q0[j], q1[j], q2[j]);
        }
    }
}

// Displacement control from the node's side: for each axis whose last-writer
// claim (list position + 1, dc_claim) is set, the claiming platen particle's
// velocity v, momentum m v and zero force.
template <typename T>
__device__ __forceinline__ void node_dc_regs(const unsigned own[3], const unsigned* __restrict__ dclist,
                                             const T* pvel, long long np, T m, T v[3], bool vset[3],
                                             T p[3], bool fzero[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!own[a]) continue;
        const T vp = pvel[a * np + dclist[own[a] - 1]];
        v[a] = vp;
        vset[a] = true;
        p[a] = m * vp;
        fzero[a] = true;
    }
}

// The node work between P2G and pass 1, one pass over the active nodes with
// the node's values in registers: displacement control (non-contact: before
// the update, …MPLocks.cpp:143-174), the grid update (IntegrateGrid, :90-142;
// contact :242-277), displacement control (contact: after it), then the
// record (f/m, m > m_min), G2P pass 1's increment (:508; FP64 form: with the
// factor dt, record_dt).  The updated momentum and the mass also go to the
// record's second half for phase B (which overwrites it with p/m and v); clean (not an output step): the
// node's mass, momentum and force are zeroed here, for the next step's P2G.
//
// work (when given): the step's boundary work in FP64, added to work[0]
// (displacement control) and work[1] (friction).  No counterpart in the
// reference, whose energy report has no external-work term
// (PhysicsEngine.cpp:140-156).  A displacement-controlled node axis takes the
// platen's velocity v and its force f is zeroed (…MPLocks.cpp:143-174;
// contact …_Contact.cpp:283-297), so the platen supplies -f there; the
// velocity field pass 2 strains the particles with is v at that node, so the
// platen's work is -f v dt.  A friction law adds df to a tangent force, whose
// work is df (p/m) dt at the updated momentum.  Summed per node in the
// form's type, per thread in double, then over the warp and added once.
template <typename T>
__device__ __forceinline__ void work_add(double* work, double w_dc, double w_fr, double dt) {
    if (!work || !__any_sync(FULL_MASK, w_dc != 0.0 || w_fr != 0.0)) return;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        w_dc += __shfl_down_sync(FULL_MASK, w_dc, off);
        w_fr += __shfl_down_sync(FULL_MASK, w_fr, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (w_dc != 0.0) atomicAdd(work, w_dc * dt);
        if (w_fr != 0.0) atomicAdd(work + 1, w_fr * dt);
    }
}

template <typename T>
__device__ __forceinline__ double dc_power(const T f[3], const T v[3], const bool fz[3]) {
    T s = (T)0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        if (fz[c]) s -= f[c] * v[c];
    return fps_f2d_form(s);
}

// FP64: small blocks, as the phases are bound by the FP64 pipe of each SM and what
// counts is that every SM gets its share of the warps.  256 / 128 / 64 / 32
// threads: 26.4 / 24.8 / 23.9 / 23.2 us (phase b 26.4 / 23.5 / 22.9 / 23.4) on
// 406k particles of honeycombs; 40k and 1k particles, whose nodes fill 35 and 3
// blocks of 256 threads, 70 -> 67 and 70 -> 65 us per step.  FP32: with 64
// threads phase b takes 16.5 us for 14.9 on the 1.89M-particle foam.
// FP32, 1280 threads per SM (phase b 1536; 1024 before): the nodes' gathers and
// records are latency and traffic, so resident warps count until registers
// spill.  5.08M-particle batch: 45.4 / 45.0 / 47.8 / 65.5 us with 1024 / 1280 /
// 1536 / 2048, phase b 40.9 / 37.9 / 35.6 / 47.3; foam 18.4 / 17.2 / 19.5 / 24.7
// and 17.7 / 16.1 / 15.9 / 21.6.
template <typename T>
constexpr int NODE_THREADS = sizeof(T) == 8 ? 64 : 256;
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 5 : 4) k_node_phase_a(NView<T> nd, T dt, double damping, int contact, int floor_friction,
                               const unsigned* __restrict__ dclist, int ndc, const T* pvel, long long np,
                               T mass_min, int clean, double* work, double dtd) {
    step_enter<sizeof(T) == 4>();
    const long long nn = nd.nn;
    double w_dc = 0.0, w_fr = 0.0;
    NODE_LOOP_AHEAD(nd, i) {
        const unsigned st = nd.state[i];
        if (!nd.alist && !(st & 1u)) continue;  // the list holds active nodes only
        const Quad<T> a0 = ld_quad(nd.acc + 8 * i), a1 = ld_quad(nd.acc + 8 * i + 4);
        const T m = a0.x;
        T p[3] = {a0.y, a0.z, a0.w}, f[3] = {a1.x, a1.y, a1.z}, v[3] = {0, 0, 0};
        const unsigned fx = nd.fixed[i];
        unsigned own[3] = {0u, 0u, 0u};
        if (ndc && (st & NODE_CLAIMED)) {
            // contact: every controlled particle claims all three axes, so one claim word serves them
#pragma unroll
            for (int a = 0; a < 3; ++a) own[a] = (contact && a > 0) ? own[0] : nd.owner[a * nn + i];
        }
        bool vset[3] = {false, false, false}, fz[3] = {false, false, false};
        if (!contact) {
            node_dc_regs<T>(own, dclist, pvel, np, m, v, vset, p, fz);
            if (work && (fz[0] | fz[1] | fz[2])) w_dc += dc_power<T>(f, v, fz);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (fz[c]) f[c] = (T)0;
        bool zero[3];
        T ft_y, dfr[3];
        grid_update_regs<T>(nd, i, fx, p, f, dt, damping, contact, floor_friction, zero, ft_y, dfr);
        if (work && (dfr[0] != (T)0 || dfr[1] != (T)0) && m > mass_min)
            w_fr += fps_f2d_form((dfr[0] * p[0] + dfr[1] * p[1]) / m);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (zero[c]) {
                v[c] = (T)0;
                vset[c] = true;
            }
            fz[c] = false;
        }
        if (contact) {
            node_dc_regs<T>(own, dclist, pvel, np, m, v, vset, p, fz);
            if (work && (fz[0] | fz[1] | fz[2])) w_dc += dc_power<T>(f, v, fz);
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (fz[c]) f[c] = (T)0;
        }
        {
            const Quad<T> w0{clean ? (T)0 : m, clean ? (T)0 : p[0], clean ? (T)0 : p[1], clean ? (T)0 : p[2]};
            const Quad<T> w1{clean ? (T)0 : f[0], clean ? (T)0 : f[1], clean ? (T)0 : f[2], (T)0};
            *reinterpret_cast<Quad<T>*>(nd.acc + 8 * i) = w0;
            *reinterpret_cast<Quad<T>*>(nd.acc + 8 * i + 4) = w1;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (vset[c]) nd.vel[c * nn + i] = v[c];
        if (fx & 2u) nd.ftemp[nn + i] += ft_y;
        const bool has = m > mass_min;
        Quad<T> r, pm;
        r.x = has ? record_dt(f[0] / m, dt) : (T)0;
        r.y = has ? record_dt(f[1] / m, dt) : (T)0;
        r.z = has ? record_dt(f[2] / m, dt) : (T)0;
        r.w = has ? (T)1 : (T)0;
        pm.x = p[0];
        pm.y = p[1];
        pm.z = p[2];
        pm.w = m;
        *reinterpret_cast<Quad<T>*>(nd.rec + 8 * i) = r;
        *reinterpret_cast<Quad<T>*>(nd.rec + 8 * i + 4) = pm;
        *reinterpret_cast<Quad<T>*>(nd.q + 4 * i) = Quad<T>{(T)0, (T)0, (T)0, (T)0};  // for pass 1's remap sums
    }
    work_add<T>(work, w_dc, w_fr, dtd);
}

// The node work between pass 1 and pass 2, in registers: the remap v += q/m
// (:559-560; phase A cleared q before pass 1 summed it), displacement
// control and BC (:573-599) in the path's order, then the record (p/m,
// m > m_min, v; FP64 form: both with the factor dt).  The claims are cleared after this last use (every claimed
// node is active: platen particles take part in P2G).  clean: a step whose
// node values nobody sees (not the last of an advance; pass 2 reads only the
// records) leaves the node zeroed as the next step's grid reset would
// (ResetGrid, …MPLocks.cpp:4-22), so that step needs no reset pass.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 6 : 4) k_node_phase_b(NView<T> nd, T dt, int contact, const unsigned* __restrict__ dclist, int ndc,
                               const T* pvel, long long np, T mass_min, int clean, int vel_zero) {
    step_enter<sizeof(T) == 4>();
    const long long nn = nd.nn;
    NODE_LOOP_AHEAD(nd, i) {
        const unsigned st = nd.state[i];
        if (!nd.alist && !(st & 1u)) continue;  // the list holds active nodes only
        const Quad<T> pm = ld_quad(nd.rec + 8 * i + 4);  // phase A's momentum and mass
        const T m = pm.w;
        const bool has = m > mass_min;
        const unsigned fx = nd.fixed[i];
        // vel_zero: the step began from a grid whose every nonzero node was in
        // the last active list (not an upload), so a node's velocity is zero
        // here unless phase A set it, which it does on fixed or claimed nodes only
        const bool vel_set = !vel_zero || fx != 0u || (st & NODE_CLAIMED);
        T v[3], p[3] = {pm.x, pm.y, pm.z};
        const Quad<T> q4 = ld_quad(nd.q + 4 * i);  // cleared by phase A, summed by pass 1
        const T q[3] = {q4.x, q4.y, q4.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = vel_set ? nd.vel[c * nn + i] : (T)0;
            if (has) v[c] = v[c] + q[c] / m;
        }
        unsigned own[3] = {0u, 0u, 0u};
        if (ndc && (st & NODE_CLAIMED)) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (contact && a > 0) {  // one claim word for the three axes (dc_claim)
                    own[a] = own[0];
                    continue;
                }
                own[a] = nd.owner[a * nn + i];
                if (own[a]) nd.owner[a * nn + i] = 0u;  // the claims' last use this step: clean for the next
            }
        }
        bool vset[3] = {false, false, false}, fz[3] = {false, false, false};
        if (!contact) node_dc_regs<T>(own, dclist, pvel, np, m, v, vset, p, fz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (fx & (1u << c)) {
                v[c] = (T)0;
                p[c] = (T)0;
                fz[c] = true;
            }
        }
        if (contact) node_dc_regs<T>(own, dclist, pvel, np, m, v, vset, p, fz);
        Quad<T> r, vq;
        r.x = has ? record_dt(p[0] / m, dt) : (T)0;
        r.y = has ? record_dt(p[1] / m, dt) : (T)0;
        r.z = has ? record_dt(p[2] / m, dt) : (T)0;
        r.w = has ? (T)1 : (T)0;
        vq.x = record_dt(v[0], dt);
        vq.y = record_dt(v[1], dt);
        vq.z = record_dt(v[2], dt);
        vq.w = (T)0;
        *reinterpret_cast<Quad<T>*>(nd.rec + 8 * i) = r;
        *reinterpret_cast<Quad<T>*>(nd.rec + 8 * i + 4) = vq;
        if (clean) {  // phase A zeroed mass, momentum and force
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (vel_set) nd.vel[c * nn + i] = (T)0;
            if (fx & 2u) nd.ftemp[nn + i] = (T)0;  // the only reaction-force entry a step writes
            nd.state[i] = contact ? 0u : (st & ~(1u | NODE_CLAIMED));
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                nd.vel[c * nn + i] = v[c];
                nd.acc[8 * i + 1 + c] = p[c];
                if (fz[c]) nd.acc[8 * i + 4 + c] = (T)0;
            }
            if (st & NODE_CLAIMED) nd.state[i] = st & ~NODE_CLAIMED;
        }
    }
}

// TimeLine::getVelocity (TimeLine.h:33-46) is evaluated on the host each step
// and passed in as tv.
struct StepArgs {
    double dt;
    float dt_f;  // RN32(dt)
    double tv[3];
    const double* tv_dev;  // graph replay: the timeline velocity computed on the device (else tv)
    int has_timeline;
    int contact;
    // return-map network (FP32 form): materials it stands in for (bit per
    // material index), the fallback half-width (fraction of k0), the queue
    int sg_on;
    unsigned sg_mats;
    float sg_band;
    SurrogateQueue q;
    SurrogateAcc* sg_acc;
    // FP32 form: von Mises hardening particles whose trial yield function is
    // above -fb_below x k0 and that the network does not take (the states at
    // and past the yield surface, and elastic ones just below it, whose
    // elastic/plastic decision FP32 rounding could flip) run the map in pairs of
    // floats (cr_increment_pairs), whose outputs are those of FP64 rounded to
    // float.  Further below the surface the map is D de, which FP32 gives to
    // within an ulp of the FP64 value rounded.
    int fb_wide;
    float fb_below;
    // harvesting of return-map inputs (either form)
    int hv_on;
    unsigned hv_mats;
    float hv_band;
    float* hv_rows;
    unsigned* hv_count;
    long long hv_cap;
    // 1: also write the step's output-only particle field (the contact path's
    // strain rate, …_Contact.cpp:509, which no later step reads), as on the
    // last step of an advance
    int outputs;
};

// The cell keys pass 2 reads and writes, by slot: this step's, the next step's
// (its sort's input, or in storage order its keys) and, on sorted steps, whose
// sort overwrites its input, a copy in slot order (`now` may be that copy;
// writing it in storage order, too, cost 20 MB a step at 5.08M particles).
struct PassKeys {
    const unsigned* now;
    unsigned* next;
    unsigned* copy;
};

// Where pass 2 reads a particle's fields from: its arrays in global memory
// (DirectSrc), or the block's copies in shared memory (StagedSrc below).
// Values written by the same step are always read back from global memory.
template <typename T>
struct DirectSrc {
    __device__ __forceinline__ unsigned pflags(const PView<T>& P, long long p) const { return P.pflags[p]; }
    __device__ __forceinline__ unsigned sid(const PView<T>& P, long long p) const { return P.sid[p]; }
    __device__ __forceinline__ unsigned key(const unsigned* keys, long long p) const { return keys[p]; }
    __device__ __forceinline__ int material(const PView<T>& P, long long p) const { return P.material[p]; }
    __device__ __forceinline__ T vol0(const PView<T>& P, long long p) const { return P.vol0[p]; }
    __device__ __forceinline__ T backstress(const PView<T>& P, long long p) const { return P.backstress[p]; }
    __device__ __forceinline__ float loc(const PView<T>& P, int k, long long p) const { return P.loc[k * P.n + p]; }
    __device__ __forceinline__ T F(const PView<T>& P, int k, long long p) const { return P.F[k * P.n + p]; }
    __device__ __forceinline__ T stress(const PView<T>& P, int k, long long p) const { return P.stress[k * P.n + p]; }
    __device__ __forceinline__ double pos(const PView<T>& P, int k, long long p) const { return P.pos[k * P.n + p]; }
};

__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait for an mbarrier phase: false, with the error bit set, when it
// does not complete within 2^22 polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned* err) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    atomicOr(err, ERR_WAIT_TIMEOUT);
    return false;
}

// The FP32 pass 2's particle fields for one block of BS particles [p0, p0 + BS)
// in shared memory, brought in by bulk copies (cp.async.bulk) that all start
// at once and complete on one mbarrier, so the block's particle reads wait
// for one memory round trip instead of one per dependent load.  One segment
// per (field, component): BS elements plus 16 bytes, copied from the 16-byte
// boundary at or below the block's first element (component k of an n-element
// array starts (k n es) mod 16 bytes into its segment).  Every array starts on
// a 16-byte boundary (cudaMalloc) and is allocated PARTICLE_PAD bytes longer
// than its n elements, so the last block's copies, which reach up to BS
// elements plus 16 bytes past the end of a component, stay inside.
constexpr size_t PARTICLE_PAD = 512 * 8 + 16;  // the largest block's elements of the widest type, and 16 bytes

template <int BS>
struct Pass2Stage {
    static_assert((size_t)BS * 8 + 16 <= PARTICLE_PAD, "padding of the particle arrays");
    static constexpr int SEG1 = BS + 16, SEG2 = 2 * BS + 16, SEG4 = 4 * BS + 16, SEG8 = 8 * BS + 16;
    static constexpr int O_FLAGS = 0, O_SID = O_FLAGS + SEG1, O_KEYS = O_SID + SEG2, O_MAT = O_KEYS + SEG4;
    static constexpr int O_VOL0 = O_MAT + SEG4, O_BACK = O_VOL0 + SEG4, O_LOC = O_BACK + SEG4;
    static constexpr int O_F = O_LOC + 3 * SEG4, O_STRESS = O_F + 9 * SEG4;
    static constexpr int O_POS = O_STRESS + 6 * SEG4, BYTES = O_POS + 3 * SEG8;
    static constexpr int NSEG = 27;  // flags, sid, keys, material, vol0, back stress, 3 loc, 9 F, 6 stress, 3 pos
    static constexpr int SMEM = BYTES + 16;  // and the mbarrier

    // segment i: its array, element size, component and shared offset
    static __device__ __forceinline__ void segment(int i, const PView<float>& P, const unsigned* keys, const void*& base,
                                                   int& es, int& k, int& off) {
        k = 0;
        if (i == 0) { base = P.pflags; es = 1; off = O_FLAGS; }
        else if (i == 1) { base = P.sid; es = 2; off = O_SID; }
        else if (i == 2) { base = keys; es = 4; off = O_KEYS; }
        else if (i == 3) { base = P.material; es = 4; off = O_MAT; }
        else if (i == 4) { base = P.vol0; es = 4; off = O_VOL0; }
        else if (i == 5) { base = P.backstress; es = 4; off = O_BACK; }
        else if (i < 9) { base = P.loc; es = 4; k = i - 6; off = O_LOC; }
        else if (i < 18) { base = P.F; es = 4; k = i - 9; off = O_F; }
        else if (i < 24) { base = P.stress; es = 4; k = i - 18; off = O_STRESS; }
        else { base = P.pos; es = 8; k = i - 24; off = O_POS; }
        off += k * (BS * es + 16);
    }
    // bytes the block's copies deliver (no specimen ids with one specimen)
    static __device__ __forceinline__ unsigned tx_bytes(const PView<float>& P) {
        return (unsigned)(BYTES - (P.sid ? 0 : SEG2));
    }
    // issue segment i's copy (called by the lanes of one warp)
    static __device__ __forceinline__ void copy(int i, const PView<float>& P, const unsigned* keys, long long p0,
                                                unsigned char* sm, uint32_t bar) {
        const void* base;
        int es, k, off;
        segment(i, P, keys, base, es, k, off);
        if (!base) return;
        const unsigned long long src = ((unsigned long long)base + (unsigned long long)(k * P.n + p0) * es) & ~15ull;
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                shared_addr(sm + off)),
            "l"(src), "r"((unsigned)(BS * es + 16)), "r"(bar)
            : "memory");
    }
};

// Reads from a Pass2Stage: thread t's element of component k sits (k n es) mod
// 16 bytes plus t es into the component's segment.
template <int BS>
struct StagedSrc {
    using S = Pass2Stage<BS>;
    const unsigned char* sm;
    template <typename E, int OFF, int ES>
    __device__ __forceinline__ E at(const PView<float>& P, int k) const {
        const unsigned mis = ((unsigned)k * (unsigned)(P.n * ES)) & 15u;
        return *reinterpret_cast<const E*>(sm + OFF + k * (BS * ES + 16) + mis + threadIdx.x * ES);
    }
    __device__ __forceinline__ unsigned pflags(const PView<float>&, long long) const { return sm[S::O_FLAGS + threadIdx.x]; }
    __device__ __forceinline__ unsigned sid(const PView<float>& P, long long) const { return at<uint16_t, S::O_SID, 2>(P, 0); }
    __device__ __forceinline__ unsigned key(const unsigned*, long long) const {
        return *reinterpret_cast<const unsigned*>(sm + S::O_KEYS + 4 * threadIdx.x);
    }
    __device__ __forceinline__ int material(const PView<float>& P, long long) const { return at<int, S::O_MAT, 4>(P, 0); }
    __device__ __forceinline__ float vol0(const PView<float>& P, long long) const { return at<float, S::O_VOL0, 4>(P, 0); }
    __device__ __forceinline__ float backstress(const PView<float>& P, long long) const {
        return at<float, S::O_BACK, 4>(P, 0);
    }
    __device__ __forceinline__ float loc(const PView<float>& P, int k, long long) const { return at<float, S::O_LOC, 4>(P, k); }
    __device__ __forceinline__ float F(const PView<float>& P, int k, long long) const { return at<float, S::O_F, 4>(P, k); }
    __device__ __forceinline__ float stress(const PView<float>& P, int k, long long) const {
        return at<float, S::O_STRESS, 4>(P, k);
    }
    __device__ __forceinline__ double pos(const PView<float>& P, int k, long long) const {
        return at<double, S::O_POS, 8>(P, k);
    }
};

// Apply a constitutive increment o to particle p (stress, plastic strain,
// back stress, energies; …MPLocks.cpp:246-270, contact …_Contact.cpp:486-525).
// The step's energy increments are summed in the form's type and added once
// to the FP64 energy accumulators.  An elastic increment (plastic = false)
// leaves the plastic strain, the plastic energy and the back stress as they
// are: they are neither read nor written (68 of the FP32 form's 324 bytes per
// particle).
// Sums that nothing in the step reads back (plastic strain and energy, on the
// contact path the strain energy, in pass 2 the strain) are added by
// reductions: the value is neither waited for nor held, and the FP64 form
// saves its FP64 pipe the addition.
template <typename T>
__device__ __forceinline__ void apply_increment(const PView<T>& P, long long p, const T sig[6], const T e[6],
                                                const CrOut<T>& o, T V, T R, bool plastic, bool contact, double dt) {
    const long long np = P.n;
    T dEs = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const T sn = sig[k] + o.dsig[k];
        P.stress[k * np + p] = sn;
        dEs += (contact ? sn : sn - (T)0.5 * o.dsig[k]) * e[k];
    }
    if (contact) {
        atomicAdd(&P.e_strain[p], fps_f2d_form(dEs * V));
    } else {
        const double es = P.e_strain[p] + fps_f2d_form(dEs * V);
        P.e_strain[p] = es;
        P.e_strain_ti[p] += es * dt;
        if (es > P.e_strain_max[p]) P.e_strain_max[p] = es;
    }
    if (!plastic) return;
    T dEp = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const T sn = sig[k] + o.dsig[k];
        atomicAdd(&P.eps_p[k * np + p], o.deps_p[k]);
        dEp += (contact ? sn : sn - (T)0.5 * o.dsig[k]) * o.deps_p[k];
    }
    atomicAdd(&P.e_plastic[p], fps_f2d_form(dEp * V));
    P.backstress[p] = R + o.dR;
}

// Trial yield function of the von Mises hardening map (…_VonMisesHardening.cpp:20-46):
// sqrt(J2) of the elastic trial stress minus the radius k0 + R/sqrt 2.
template <typename T>
__device__ __forceinline__ T vmh_trial(const MatConst& m, T R, const T sig[6], const T e[6]) {
    T d[6];
    trial_increment<T>(m, e, d);
    T tr[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) tr[i] = sig[i] + d[i];
    const T a01 = tr[0] - tr[1], a12 = tr[1] - tr[2], a20 = tr[2] - tr[0];
    T J2 = (T)(1.0 / 6.0) * a01 * a01;
    J2 += (T)(1.0 / 6.0) * a12 * a12;
    J2 += (T)(1.0 / 6.0) * a20 * a20;
    J2 += tr[3] * tr[3];
    J2 += tr[4] * tr[4];
    J2 += tr[5] * tr[5];
    return sqrt(J2) - (form_const<T>(m.k0, m.fk0) + R * (T)0.70710678118654752440);
}

// warp-aggregated increment of a device counter; returns this lane's slot
__device__ __forceinline__ unsigned warp_slot(unsigned* counter) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned)__popc(m));
    base = __shfl_sync(m, base, leader);
    return base + __popc(m & ((1u << lane) - 1u));
}

// The particle arrays pass 2 reads, one per thread of a block's first warps:
// prefetched into L2 for the block's particle range while the warps gather
// the node records.
template <typename T>
__device__ __forceinline__ void pass2_prefetch(const PView<T>& P, long long p0, int cnt, int contact) {
    const int t = threadIdx.x;
    const long long n = P.n;
    const void* base = nullptr;
    int es = (int)sizeof(T);
    long long comp = 0;
    if (t < 3) {
        base = P.pos;
        es = 8;
        comp = t;
    } else if (t < 12) {
        base = P.F;
        comp = t - 3;
    } else if (t < 18) {
        base = P.stress;
        comp = t - 12;
    } else if (t == 18) {
        base = P.vol0;
    } else if (t == 19) {
        base = P.backstress;
    } else if (t == 20) {
        base = P.material;
        es = 4;
    } else if (t == 21) {
        base = P.pflags;
        es = 1;
    } else if (t == 22 && !contact) {
        base = P.e_strain;
        es = 8;
    } else if (t == 23 && !contact) {
        base = P.e_strain_ti;
        es = 8;
    } else if (t == 24 && !contact) {
        base = P.e_strain_max;
        es = 8;
    }
    if (base) prefetch_l2((const char*)base + comp * n * es, es, n, p0, cnt);
}

// ---------------------------------------------------------------------------
// G2P pass 2 + constitutive update + platen (G2P_P2_SmallStrain,
// …MPLocks.cpp:175-280; contact …_Contact.cpp:438-525 and :531-540).
// One thread per particle in index order (coalesced particle streams).  At
// the end each particle also computes the cell key (and, in the FP32 form,
// the cell-local coordinate) of its new position for the next step, so the
// next step needs no separate key pass.
// ---------------------------------------------------------------------------
// The large-strain pass 2's update of one particle after its gather
// (G2P_P2_LargeStrain, …MPLocks.cpp:311-435; FP64 form): the stress is reset,
// the logarithmic strains of F F^T (total, from the old F), of the trial
// elastic gradient dF F_e and of the increment dF are formed, the
// constitutive map takes zero stress and the trial elastic strain and returns
// the Kirchhoff stress, F_e becomes the exponential of the elastic strain,
// F = F dF, and stress = Kirchhoff / det F.  Energies add stress x increment x
// V component by component, as the reference does.
template <typename T>
__device__ __forceinline__ void large_strain_update(const PView<T>& P, long long p, const T Ldt[9],
                                                    const MatConst* __restrict__ mats, int nmat, unsigned* err) {
    if constexpr (sizeof(T) == 8) {
        const long long np = P.n;
#pragma unroll
        for (int k = 0; k < 6; ++k) P.stress[k * np + p] = 0.0;
        double dF[9], F[9], Fe[9];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) dF[3 * c + r] = (c == r ? 1.0 : 0.0) + (double)Ldt[3 * c + r];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            F[k] = P.F[k * np + p];
            Fe[k] = P.Fe[k * np + p];
        }
        double et[6], ee[6], einc[6], Fet[9];
        half_log_voigt(F, et);
        mat3_mul(dF, Fe, Fet);
        half_log_voigt(Fet, ee);
        half_log_voigt(dF, einc);
        const int mi = P.material[p];
        if (!(mi >= 0 && mi < nmat)) {
            atomicOr(err, ERR_BAD_MATERIAL);
            return;
        }
        const double zero[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        CrOut<double> o;
        cr_increment<double>(mats[mi], (double)P.backstress[p], zero, ee, o);
        double el[6], E[9], Fen[9], Fn[9];
#pragma unroll
        for (int k = 0; k < 6; ++k) el[k] = ee[k] - o.deps_p[k];
        E[0] = el[0];
        E[4] = el[1];
        E[8] = el[2];
        E[1] = E[3] = 0.5 * el[3];
        E[5] = E[7] = 0.5 * el[4];
        E[2] = E[6] = 0.5 * el[5];
        mat3_exp8(E, Fen);
        mat3_mul(F, dF, Fn);
        const double det = Kinematics<double>::det(Fn);
        const double V = det * (double)P.vol0[p];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            P.Fe[k * np + p] = Fen[k];
            P.F[k * np + p] = Fn[k];
        }
        P.vol[p] = V;
        double es = P.e_strain[p], ep = P.e_plastic[p];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double sn = (1.0 / det) * o.dsig[k];
            P.strain[k * np + p] = et[k];
            P.stress[k * np + p] = sn;
            atomicAdd(&P.eps_p[k * np + p], o.deps_p[k]);
            es += sn * einc[k] * V;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) ep += (1.0 / det) * o.dsig[k] * o.deps_p[k] * V;
        P.e_strain[p] = es;
        P.e_plastic[p] = ep;
        P.backstress[p] += o.dR;
    }
}

// One particle of pass 2; returns the new cell key (u: the new cell-local
// coordinate; queued: its stress increment waits for the network).
template <typename T, int BATCH, bool CONTACT, bool LS = false, class SRC = DirectSrc<T>>
__device__ __forceinline__ unsigned pass2_particle(const PView<T>& P, const NView<T>& nd, const Geom& g,
                                                   const PassKeys& keys, const MatConst* __restrict__ mats, int nmat,
                                                   const StepArgs& a, unsigned* err, long long p, float u[3],
                                                   bool& queued, const SRC& src = SRC{}) {
    const long long np = P.n;
    queued = false;
    const unsigned fl = src.pflags(P, p);
    const T dt = form_const<T>(a.dt, a.dt_f);
    const bool skip = CONTACT && (fl & 8u);
    const Geom& gs = (g.nspec > 1) ? g.tab[src.sid(P, p)] : g;
    // the position stays in registers until the new cell key is formed
    double x[3] = {src.pos(P, 0, p), src.pos(P, 1, p), src.pos(P, 2, p)};
    if (!skip) {
        const unsigned key = src.key(keys.now, p);
        T Ldt[9];  // velocity gradient times dt
#pragma unroll
        for (int k = 0; k < 9; ++k) Ldt[k] = 0;
        if (key < g.key_max) {
            int b[3];
            key_to_base(key, gs, b);
            Bases<T> B;
            if constexpr (sizeof(T) == 4) {
                const float ul[3] = {src.loc(P, 0, p), src.loc(P, 1, p), src.loc(P, 2, p)};
                B.init_local(gs, ul);
            } else {
                particle_bases<T>(P, gs, p, b, B);
            }
            // An (x, y) pair of corners shares A = Nx Ny, Bx = Ny gx and By =
            // Nx gy; a record's r is zero where m <= mass_min, and grad N =
            // -(Bx Nz, By Nz, A gz).
            // FP32 form: displacement and L are summed corner by corner, the
            // records hold p/m and v, and dt comes last, per particle.  Other
            // orders have the same number of roundings, but some that do not
            // change from step to step: with dt taken per node and the pair
            // summed along z first, 99% of the positions of 300k particles
            // in three materials stayed within 2.9e-9 h of corner order's
            // after 120 steps, where two runs of one code stay within 1.1e-9
            // (1.07M block 6.4e-10 and 4.7e-10, honeycombs 5.1M 3.4e-10 and
            // 1.8e-10), and the error against the FP64 form grew by 1.4 to
            // 1.6.  Corner order and dt here cost 2% (honeycombs 685 us per
            // step, 668 the other way).
            // FP64 form (bound by its FP64 pipe): the records carry dt; L is
            // summed along z first,
            //   L_x -= Bx (Nz v), L_y -= By (Nz v), L_z -= A (gz v),
            // 132 products and sums per particle instead of 168; the position
            // is added to per corner in the reference's order
            // (…MPLocks.cpp:197-198), so it keeps its last bits, on which the
            // ties of the contact normals turn.
            T disp[3] = {0, 0, 0};
            const CellNodes cn = cell_nodes(gs, b);
#pragma unroll(sizeof(T) == 4 ? 4 : (BATCH ? 2 : 1))
            for (int h = 0; h < 4; ++h) {
                Quad<T> rq[2], vq[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const Quad<T> z{(T)0, (T)0, (T)0, (T)0};
                    rq[j] = z;
                    vq[j] = z;
                    if ((cn.mask >> (2 * h + j)) & 1u) ld_record(nd.rec + 8ll * cell_node(cn, 2 * h + j), rq[j], vq[j]);
                }
                const bool ix = (h >> 1) & 1, iy = h & 1;
                const T nx = ix ? B.Nx[1] : B.Nx[0], ny = iy ? B.Ny[1] : B.Ny[0];
                const T gx = ix ? B.gx[1] : B.gx[0], gy = iy ? B.gy[1] : B.gy[0], A = nx * ny;
                const T r0[3] = {rq[0].x, rq[0].y, rq[0].z}, r1[3] = {rq[1].x, rq[1].y, rq[1].z};
                const T v0[3] = {vq[0].x, vq[0].y, vq[0].z}, v1[3] = {vq[1].x, vq[1].y, vq[1].z};
                // outerProduct(v_i, grad N): column c, row r = v_i[r] * G[c]
                if constexpr (sizeof(T) == 4) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float nz = B.Nz[j], N = A * nz;
                        const float Gx = -(ny * nz) * gx, Gy = -(nx * nz) * gy, Gz = -A * B.gz[j];
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float v = j ? v1[c] : v0[c];
                            disp[c] += N * (j ? r1[c] : r0[c]);
                            Ldt[c] += v * Gx;
                            Ldt[3 + c] += v * Gy;
                            Ldt[6 + c] += v * Gz;
                        }
                    }
                } else {
                    const double Bx = ny * gx, By = nx * gy;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double w = B.Nz[0] * v0[c] + B.Nz[1] * v1[c], d = B.gz[0] * v0[c] + B.gz[1] * v1[c];
                        x[c] = x[c] + A * B.Nz[0] * r0[c];
                        x[c] = x[c] + A * B.Nz[1] * r1[c];
                        Ldt[c] -= Bx * w;
                        Ldt[3 + c] -= By * w;
                        Ldt[6 + c] -= A * d;
                    }
                }
            }
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int c = 0; c < 3; ++c) x[c] += fps_f2d(disp[c] * dt);
#pragma unroll
                for (int k = 0; k < 9; ++k) Ldt[k] *= dt;
            }
        }
        if constexpr (LS) {
            large_strain_update(P, p, Ldt, mats, nmat, err);
        } else {
        // strain increment: diagonal from dF = I + L dt (form-specific, see
        // Kinematics), off-diagonal (L_ij + L_ji) dt in Voigt engineering shear
        T e[6];
        e[0] = Kinematics<T>::strain_diag(Ldt[0]);
        e[1] = Kinematics<T>::strain_diag(Ldt[4]);
        e[2] = Kinematics<T>::strain_diag(Ldt[8]);
        e[3] = Ldt[1] + Ldt[3];
        e[4] = Ldt[5] + Ldt[7];
        e[5] = Ldt[6] + Ldt[2];
        const int mi = src.material(P, p);
        const bool have_mat = mi >= 0 && mi < nmat;
        T V = 0;
        // strain, F and V: on the contact path before the material check
        // (…_Contact.cpp:464-484), else with a material only (…MPLocks.cpp:226-258)
        if (CONTACT || have_mat) {
            T F[9], Fn[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) F[k] = src.F(P, k, p);
            Kinematics<T>::update(CONTACT, F, Ldt, Fn);
#pragma unroll
            for (int k = 0; k < 9; ++k) P.F[k * np + p] = Fn[k];
            V = Kinematics<T>::det(Fn) * src.vol0(P, p);
            P.vol[p] = V;
#pragma unroll
            for (int k = 0; k < 6; ++k) atomicAdd(&P.strain[k * np + p], e[k]);
        }
        if (have_mat) {
            const MatConst& M = mats[mi];
            if (CONTACT && a.outputs) {
#pragma unroll
                for (int k = 0; k < 6; ++k) P.strain_rate[k * np + p] = e[k] / dt;
            }
            T sig[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) sig[k] = src.stress(P, k, p);
            const T R = src.backstress(P, p);
            CrOut<T> o;
            // the network takes clearly plastic trial states of the materials it
            // was trained for; the band near the surface and elastic states stay
            // exact, the band (and every plastic state the network does not take)
            // by the map in pairs of floats
            CrTrial<T> tr;
            cr_trial<T>(M, R, sig, e, tr);
            bool wide = false, plastic = false;
            if constexpr (sizeof(T) == 4) {
                if (M.type == 4) {
                    const float f = sqrtf(tr.J2) - tr.rad;  // the trial yield function (…_VonMisesHardening.cpp:35-46)
                    if (a.sg_on && mi < 32 && ((a.sg_mats >> mi) & 1u)) {
                        queued = f >= a.sg_band * M.fk0;
                        if (!queued && f > 0.0f) {
                            const unsigned m = __activemask();
                            if ((threadIdx.x & 31) == __ffs(m) - 1) atomicAdd(&a.sg_acc->band, (unsigned long long)__popc(m));
                        }
                    }
                    wide = a.fb_wide && !queued && f > -a.fb_below * M.fk0;
                }
            }
            if (a.hv_on && mi < 32 && ((a.hv_mats >> mi) & 1u) && M.type == 4 &&
                vmh_trial<T>(M, R, sig, e) >= (T)a.hv_band * form_const<T>(M.k0, M.fk0)) {
                const unsigned slot = warp_slot(a.hv_count);
                if (slot < (unsigned long long)a.hv_cap) {
                    float* hr = a.hv_rows + (long long)slot * 13;
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        hr[k] = (float)sig[k];
                        hr[7 + k] = (float)e[k];
                    }
                    hr[6] = (float)R;
                }
            }
            if (queued) {
                if constexpr (sizeof(T) == 4) {
                    const unsigned slot = warp_slot(a.q.count);
                    if (slot < (unsigned long long)a.q.cap) {
                        float* qi = a.q.in + (long long)slot * 13;
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            qi[k] = sig[k];
                            qi[7 + k] = e[k];
                        }
                        qi[6] = R;
                        a.q.vol[slot] = V;
                        a.q.pidx[slot] = (unsigned)p;
                    }
                }
            } else {
                if constexpr (sizeof(T) == 4) {
                    if (wide)
                        plastic = cr_increment_pairs(M, R, sig, e, tr, o);
                    else
                        plastic = cr_return<T>(M, R, sig, e, tr, o);
                } else {
                    plastic = cr_return<T>(M, R, sig, e, tr, o);
                }
                apply_increment<T>(P, p, sig, e, o, V, R, plastic, CONTACT, a.dt);
            }
        } else if (!CONTACT) {
            atomicOr(err, ERR_BAD_MATERIAL);
        }
        }
    }
    // platen timeline (…MPLocks.cpp:766-789; contact :531-540)
    if (fl & PF_IN_DC) {
        const double* tv = a.tv_dev ? a.tv_dev : a.tv;
        if constexpr (!CONTACT) {
            if (a.has_timeline) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (fl & (1u << c)) P.vel[c * np + p] = (T)((double)P.dc_mult[p] * tv[c]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double vv = a.has_timeline ? (double)P.dc_mult[p] * tv[c] : (double)P.vel[c * np + p];
                P.vel[c * np + p] = (T)vv;
                x[c] += vv * a.dt;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) P.pos[c * np + p] = x[c];
    // the next step's cell key (and FP32 cell-local coordinate) from the new position
    const unsigned nk = particle_key(gs, x, u, err);
    keys.next[p] = nk;
    if (keys.copy) keys.copy[p] = nk;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int c = 0; c < 3; ++c) P.loc[c * np + p] = u[c];
    }
    return nk;
}

// BS: the block size; the FP32 form asks for 1024 / BS blocks per SM (64
// registers).  Blocks of 128, us per step of a 1.07M-particle block and of 5.08M
// particles of honeycombs: 142.9 and 677 with 768 threads per SM, 140.3 and 665
// with 896, 138.4 and 657 with 1024, 140.0 and 660 with 1152; 144.6 and 679 with
// 1280 (256 threads per block; 48 registers and spills); those with the pairs of
// corners summed along z first, now 151.5 and 679 with 1024.  CONTACT: the loop's path, apart so that each kernel holds
// one path's code (pass 2's warps also wait for instructions).
template <typename T, int BATCH, int BS, bool CONTACT>
__global__ void __launch_bounds__(BS, sizeof(T) == 4 ? 1024 / BS : 1) k_pass2(PView<T> P, NView<T> nd, Geom g, PassKeys keys,
                                               const MatConst* __restrict__ mats, int nmat, StepArgs a, unsigned* err) {
    step_enter<sizeof(T) == 4>();
    const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (threadIdx.x < 32) pass2_prefetch<T>(P, blockIdx.x * (long long)blockDim.x, blockDim.x, CONTACT);
    if (p >= P.n) return;
    float u[3];
    bool queued;
    pass2_particle<T, BATCH, CONTACT>(P, nd, g, keys, mats, nmat, a, err, p, u, queued);
}

// FP32 pass 2 with the block's particle fields staged in shared memory
// (Pass2Stage): warp 0 issues the bulk copies, every thread waits once on the
// mbarrier, then runs pass2_particle reading from shared memory.  The arrays
// are allocated with room for the last block's copies (PARTICLE_PAD).
// Blocks per SM: as many as the staging buffers fit (228 KB of shared memory,
// 1 KB reserved per block), but no more than 1024 threads, which leaves 64
// registers per thread.  At 6, 7, 8, 9 and 10 blocks of 128 the step of a solid
// block of 1.07M particles in mid-crush took 147.8, 145.5, 145.8, 146.1 and
// 150.0 us, that of 5.08M particles of honeycombs 700, 691, 689, 686 and 700.
// Before the sums that nothing reads back became reductions and each path got
// a kernel of its own, 168 and 752 us (pass 2 117 and 410 us, now 89 and 342).
template <int BS>
constexpr int pass2_staged_blocks() {
    constexpr int fit = (228 * 1024) / (Pass2Stage<BS>::SMEM + 1024), want = 1024 / BS;
    return fit < want ? fit : want;
}

template <int BS, bool CONTACT>
__global__ void __launch_bounds__(BS, pass2_staged_blocks<BS>()) k_pass2_staged(PView<float> P, NView<float> nd, Geom g,
                                                               PassKeys keys, const MatConst* __restrict__ mats,
                                                               int nmat, StepArgs a, unsigned* err) {
    using S = Pass2Stage<BS>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x;
    const long long p0 = blockIdx.x * (long long)BS, p = p0 + t;
    float u[3];
    bool queued;
    const uint32_t bar = shared_addr(smem_raw + S::BYTES);
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    step_enter<true>();
    __syncthreads();
    if (t < 32) {
        if (t == 0)
            asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(bar),
                         "r"(S::tx_bytes(P))
                         : "memory");
        __syncwarp();
        if (t < S::NSEG) S::copy(t, P, keys.now, p0, smem_raw, bar);
    }
    if (!mbar_wait(bar, 0, err)) {
        mbar_wait(bar, 0, err);  // once more (bounded) for copies still in flight, then leave
        return;
    }
    if (p >= P.n) return;
    pass2_particle<float, 0, CONTACT, false, StagedSrc<BS>>(P, nd, g, keys, mats, nmat, a, err, p, u, queued,
                                                            StagedSrc<BS>{smem_raw});
}

// The large-strain pass 2 (non-contact loop, FP64 form; the reference ships
// it disabled, …MPLocks.cpp:605, and MPM_OPT_LARGE_STRAIN switches it on).
template <int BS>
__global__ void __launch_bounds__(BS) k_pass2_ls(PView<double> P, NView<double> nd, Geom g, PassKeys keys,
                                                 const MatConst* __restrict__ mats, int nmat, StepArgs a, unsigned* err) {
    step_enter<false>();
    const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p >= P.n) return;
    float u[3];
    bool queued;
    pass2_particle<double, 0, false, true>(P, nd, g, keys, mats, nmat, a, err, p, u, queued);
}

// ---------------------------------------------------------------------------
// Contact detection (…_Contact.cpp:152-237), bit-exact.
// Node mass gradients sum grad N m_p over all particles; the reference adds
// them in particle index order (one thread), and the max-norm selection that
// follows is sensitive to the last bit.  Only nodes adjacent to surface
// particles are ever read, so only those are summed here, over the particles of
// the eight surrounding cells in index order, with the reference's exact
// per-pair gradient.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_contact_need(PView<T> P, const unsigned* __restrict__ keys, Geom g, unsigned* __restrict__ need,
                               const unsigned* __restrict__ surf, int nsurf) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsurf) return;
    const long long p = surf[t];
    unsigned key = keys[p];
    if (key >= g.key_max) return;
    const Geom& gs = spec_geom(g, P.sid, p);
    int b[3];
    key_to_base(key, gs, b);
    for (int k = 0; k < 8; ++k) {
        long long nid = corner_node(gs, b, k);
        if (nid >= 0) need[nid] = 1u;
    }
}

// Compact the needed nodes into a list (order irrelevant: nodes are independent).
static __global__ void k_contact_compact(const unsigned* __restrict__ need, long long nn, unsigned* __restrict__ list,
                                         unsigned* __restrict__ count) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    bool take = i < nn && need[i];
    unsigned m = __ballot_sync(FULL_MASK, take);
    if (!m) return;
    int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned)__popc(m));
    base = __shfl_sync(m, base, leader);
    if (take) list[base + __popc(m & ((1u << lane) - 1u))] = (unsigned)i;
}

// One warp per needed node: gather the slots of the eight surrounding cells'
// particles into shared memory, rank them by the caller's particle index (the
// slot itself when particles are not stored in cell order), and compute each
// pair's exact grad N * m in parallel.  The sums in index order are serial
// chains of FP64 additions, each costing the pipe a whole warp's slot however
// few its lanes: the block's first warp adds all of the block's nodes' chains
// together, three lanes per node (one node's chain per warp before: 884 us for
// the 406k-particle honeycombs, now 439, with exact_gradient's comparisons off the pipe).
// Nodes with more than CG_CAP contributors take the selection below:
// the warp looks for the next larger index among all of them, one at a time.
constexpr int CG_WARPS = 8;
static_assert(3 * CG_WARPS <= 32, "one warp adds the block's chains");
constexpr int CG_CAP = 256;

template <typename T>
__device__ __forceinline__ unsigned caller_index(const PView<T>& P, unsigned slot) {
    return P.orig ? P.orig[slot] : slot;
}

template <typename T>
__device__ __noinline__ void mass_gradient_select(const PView<T>& P, const Geom& g, const int node[3],
                                                  const unsigned* __restrict__ perm, const unsigned seg[8],
                                                  const unsigned off[8], unsigned total, double gsum[3]) {
    const long long np = P.n;
    const int lane = threadIdx.x & 31;
    gsum[0] = gsum[1] = gsum[2] = 0.0;
    long long last = -1;
    for (unsigned done = 0; done < total; ++done) {
        unsigned best = 0xffffffffu, slot = 0;
        for (unsigned e = lane; e < total; e += 32) {
            int k = 0;
            for (int kk = 1; kk < 8; ++kk)
                if (e >= off[kk]) k = kk;
            const unsigned sl = perm[seg[k] + (e - off[k])], id = caller_index(P, sl);
            if ((long long)id > last && id < best) {
                best = id;
                slot = sl;
            }
        }
        const unsigned next = __reduce_min_sync(FULL_MASK, best);
        const unsigned from = __ballot_sync(FULL_MASK, best == next);
        slot = __shfl_sync(FULL_MASK, slot, __ffs(from) - 1);
        last = next;
        const double x[3] = {P.pos[slot], P.pos[np + slot], P.pos[2 * np + slot]};
        double G[3];
        exact_gradient(g, x, node, G);
        const double m = (double)P.mass[slot];
        for (int c = 0; c < 3; ++c) gsum[c] = __dadd_rn(gsum[c], __dmul_rn(G[c], m));
    }
}

struct ContactScratch {
    double c[CG_WARPS][CG_CAP][3];    // contributions by rank
    unsigned id[CG_WARPS][CG_CAP];    // the caller's index
    unsigned total[CG_WARPS];         // ranked contributors
    long long node[CG_WARPS];         // -1: the warp has no node, or has summed it itself
};

template <typename T>
__global__ void __launch_bounds__(CG_WARPS * 32) k_contact_mass_gradient(PView<T> P, NView<T> nd, Geom g,
                                                                         const unsigned* __restrict__ list,
                                                                         const unsigned* __restrict__ count,
                                                                         const unsigned* __restrict__ perm,
                                                                         const unsigned* __restrict__ cstart,
                                                                         const unsigned* __restrict__ cend) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ContactScratch& S = *reinterpret_cast<ContactScratch*>(smem_raw);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long np = P.n, nn = nd.nn;
    const unsigned total_nodes = *count;
    for (unsigned first = blockIdx.x * CG_WARPS; first < total_nodes; first += gridDim.x * CG_WARPS) {
        const unsigned item = first + w;
        if (lane == 0) S.node[w] = -1;
        if (item < total_nodes) {
            const long long i = list[item];
            const Geom& gs = node_geom(g, i);
            const long long il = i - gs.node_off;
            int node[3];
            node[0] = (int)(il % gs.nn[0]);
            node[1] = (int)((il / gs.nn[0]) % gs.nn[1]);
            node[2] = (int)(il / ((long long)gs.nn[0] * gs.nn[1]));
            // lanes 0..7: the eight surrounding cells (cell = node - {0,1}^3)
            unsigned s0 = 0, len = 0;
            if (lane < 8) {
                int cb[3] = {node[0] - ((lane >> 2) & 1), node[1] - ((lane >> 1) & 1), node[2] - (lane & 1)};
                unsigned key = gs.key_off + (unsigned)((cb[0] + 1) + gs.kd[0] * ((cb[1] + 1) + gs.kd[1] * (cb[2] + 1)));
                s0 = cstart[key];
                unsigned s1 = cend[key];
                len = s1 > s0 ? s1 - s0 : 0u;
            }
            // exclusive offsets of the segments
            unsigned off = len;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                unsigned o = __shfl_up_sync(FULL_MASK, off, d);
                if (lane >= d) off += o;
            }
            const unsigned total = __shfl_sync(FULL_MASK, off, 7);
            off -= len;
            unsigned segs[8], offs[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                segs[k] = __shfl_sync(FULL_MASK, s0, k);
                offs[k] = __shfl_sync(FULL_MASK, off, k);
            }
            if (total > (unsigned)CG_CAP) {
                double gsum[3] = {0.0, 0.0, 0.0};
                mass_gradient_select<T>(P, gs, node, perm, segs, offs, total, gsum);
                if (lane == 0) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) nd.mg[c * nn + i] = gsum[c];
                }
            } else {
                auto slot_of = [&](unsigned e) {
                    int k = 0;
#pragma unroll
                    for (int kk = 1; kk < 8; ++kk)
                        if (e >= offs[kk]) k = kk;
                    return perm[segs[k] + (e - offs[k])];
                };
                for (unsigned e = lane; e < total; e += 32) S.id[w][e] = caller_index(P, slot_of(e));
                __syncwarp();
                for (unsigned e = lane; e < total; e += 32) {
                    const unsigned key = S.id[w][e], id = slot_of(e);
                    unsigned rank = 0;
                    for (unsigned j = 0; j < total; ++j) rank += S.id[w][j] < key ? 1u : 0u;
                    double x[3] = {P.pos[id], P.pos[np + id], P.pos[2 * np + id]};
                    double G[3];
                    exact_gradient(gs, x, node, G);
                    const double m = (double)P.mass[id];
                    S.c[w][rank][0] = __dmul_rn(G[0], m);
                    S.c[w][rank][1] = __dmul_rn(G[1], m);
                    S.c[w][rank][2] = __dmul_rn(G[2], m);
                }
                if (lane == 0) {
                    S.node[w] = i;
                    S.total[w] = total;
                }
            }
        }
        __syncthreads();
        if (w == 0 && lane < 3 * CG_WARPS && S.node[lane / 3] >= 0) {
            const int q = lane / 3, c = lane % 3;
            double acc = 0.0;
            for (unsigned e = 0; e < S.total[q]; ++e) acc = __dadd_rn(acc, S.c[q][e][c]);
            nd.mg[c * nn + S.node[q]] = acc;
        }
        __syncthreads();
    }
}

// The contact kernels below run one thread per surface particle (a list
// compacted at upload).  FP64 form: the reference's uncontracted FP64
// arithmetic, bit-exact.  FP32 form: the same tests in FP32 (the flags only
// feed output, as in the reference, where nothing reads them back).
__device__ __forceinline__ float dot3f(const float a[3], const float b[3]) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// Surface particle normal: the corner gradient of largest norm, first wins on ties (:156-172).
template <typename T>
__global__ void k_contact_mp_gradient(PView<T> P, NView<T> nd, Geom g, const unsigned* __restrict__ keys,
                                      const unsigned* __restrict__ surf, int nsurf) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsurf) return;
    const long long p = surf[t];
    const Geom& gs = spec_geom(g, P.sid, p);
    const long long np = P.n, nn = nd.nn;
    T gp[3] = {0, 0, 0};
    unsigned key = keys[p];
    if (key < g.key_max) {
        int b[3];
        key_to_base(key, gs, b);
        float best2 = 0.0f;
        for (int k = 0; k < 8; ++k) {
            long long nid = corner_node(gs, b, k);
            if (nid < 0) continue;
            T gi[3] = {nd.mg[nid], nd.mg[nn + nid], nd.mg[2 * nn + nid]};
            bool take;
            if constexpr (sizeof(T) == 8) {
                take = len3_rn(gi) > len3_rn(gp);
            } else {
                float l2 = dot3f(gi, gi);
                take = l2 > best2;
                if (take) best2 = l2;
            }
            if (take) {
                gp[0] = gi[0];
                gp[1] = gi[1];
                gp[2] = gi[2];
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) P.mp_mg[c * np + p] = gp[c];
}

// Reset the node mass gradient of active nodes (:177-186) and the normal claims.
template <typename T>
__device__ __forceinline__ void contact_reset_node(const NView<T>& nd, long long i) {
    nd.nowner[i] = 0u;
    if (!(nd.state[i] & 1u)) return;
    const long long nn = nd.nn;
#pragma unroll
    for (int c = 0; c < 3; ++c) nd.mg[c * nn + i] = 0.0;
}

template <typename T>
__global__ void k_contact_reset(NView<T> nd) {
    NODE_LOOP(nd, i) contact_reset_node<T>(nd, i);
}

// Node normal from surface particles with (x_i - x_p) . g_p > 0 (:191-210);
// the reference overwrites in index order, so the largest index wins.
template <typename T>
__global__ void k_contact_normal(PView<T> P, NView<T> nd, Geom g, const unsigned* __restrict__ keys,
                                 const unsigned* __restrict__ surf, int nsurf, int apply) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsurf) return;
    const long long p = surf[t];
    const Geom& gs = spec_geom(g, P.sid, p);
    const long long np = P.n, nn = nd.nn;
    unsigned key = keys[p];
    if (key >= g.key_max) return;
    int b[3];
    key_to_base(key, gs, b);
    const T gp[3] = {P.mp_mg[p], P.mp_mg[np + p], P.mp_mg[2 * np + p]};
    for (int k = 0; k < 8; ++k) {
        long long nid = corner_node(gs, b, k);
        if (nid < 0) continue;
        int o3[3] = {(k >> 2) & 1, (k >> 1) & 1, k & 1};
        bool facing;
        if constexpr (sizeof(T) == 8) {
            double d[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) d[c] = __dadd_rn(node_coord(gs, c, b[c] + o3[c]), -P.pos[c * np + p]);
            facing = dot3_rn(d, gp) > 0.0;
        } else {
            // node minus particle from the cell-local coordinate: (o - u) h per axis
            float d[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) d[c] = ((float)o3[c] - P.loc[c * np + p]) * gs.hf[c];
            facing = dot3f(d, gp) > 0.0f;
        }
        if (!facing) continue;
        const unsigned who = (P.orig ? P.orig[p] : (unsigned)p) + 1u;  // the caller's particle order
        if (!apply) {
            atomicMax(&nd.nowner[nid], who);
        } else if (nd.nowner[nid] == who) {
#pragma unroll
            for (int c = 0; c < 3; ++c) nd.mg[c * nn + nid] = gp[c];
        }
    }
}

// Contact flags (:215-237): g_i . g_p >= 0.001 |g_i| |g_p| -> positive, <= -tol -> negative.
template <typename T>
__global__ void k_contact_flags(PView<T> P, NView<T> nd, Geom g, const unsigned* __restrict__ keys,
                                const unsigned* __restrict__ surf, int nsurf) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsurf) return;
    const long long p = surf[t];
    const Geom& gs = spec_geom(g, P.sid, p);
    const long long np = P.n, nn = nd.nn;
    unsigned key = keys[p];
    if (key >= g.key_max) return;
    int b[3];
    key_to_base(key, gs, b);
    const T gp[3] = {P.mp_mg[p], P.mp_mg[np + p], P.mp_mg[2 * np + p]};
    double lp = 0.0;
    float lpf = 0.0f;
    if constexpr (sizeof(T) == 8)
        lp = len3_rn(gp);
    else
        lpf = sqrtf(dot3f(gp, gp));
    for (int k = 0; k < 8; ++k) {
        long long nid = corner_node(gs, b, k);
        if (nid < 0) continue;
        const T gi[3] = {nd.mg[nid], nd.mg[nn + nid], nd.mg[2 * nn + nid]};
        bool pos, neg;
        if constexpr (sizeof(T) == 8) {
            double tol = __dmul_rn(__dmul_rn(0.001, len3_rn(gi)), lp);
            double dd = dot3_rn(gi, gp);
            pos = dd >= tol;
            neg = !pos && dd <= -tol;
        } else {
            float tol = 0.001f * sqrtf(dot3f(gi, gi)) * lpf;
            float dd = dot3f(gi, gp);
            pos = dd >= tol;
            neg = !pos && dd <= -tol;
        }
        if (pos)
            atomicOr(&nd.state[nid], 4u);
        else if (neg)
            atomicOr(&nd.state[nid], 8u);
    }
}

// ---------------------------------------------------------------------------
// Console monitors (PhysicsEngine::reportConsole, PhysicsEngine.cpp:40-183).
// acc layout (doubles): 0-2 position sum, 3-5 momentum, 6 max |principal
// strain|, 7 max |principal stress|, 8-10 stress sum, 11-13 strain sum,
// 14 kinetic, 15 strain energy, 16 plastic energy, 17-19 reaction-force sum;
// counts (u64) follow at 24-28.
// ---------------------------------------------------------------------------
constexpr int MON_SLOTS = 32;

// ConstitutiveRelation::getPrincipal (ConstitutiveRelation_calculateState.cpp:160-196),
// largest |principal value|; NaN (hydrostatic or zero states) or Q > 0 give 0,
// as the reference's max update skips them.
__device__ __forceinline__ double principal_abs_max(const double s[6]) {
    const double I1 = s[0] + s[1] + s[2];
    double I2 = 0.0;
    I2 += s[0] * s[1];
    I2 += s[1] * s[2];
    I2 += s[0] * s[2];
    I2 -= s[3] * s[3];
    I2 -= s[4] * s[4];
    I2 -= s[5] * s[5];
    // symmetric matrix [[s0 s3 s5] [s3 s1 s4] [s5 s4 s2]], glm cofactor determinant
    const double m[9] = {s[0], s[3], s[5], s[3], s[1], s[4], s[5], s[4], s[2]};
    const double I3 = Kinematics<double>::det(m);
    const double Q = (3.0 * I2 - I1 * I1) / 9.0;
    const double R = (2.0 * I1 * I1 * I1 - 9.0 * I1 * I2 + 27.0 * I3) / 54.0;
    if (Q > 0.0) return 0.0;
    double T = R / sqrt(-Q * Q * Q);
    if (!(T == T)) return 0.0;
    T = fmin(fmax(T, -1.0), 1.0);
    const double th = acos(T), pi = 3.14159265359;  // _PI, Definitions.h:12
    double best = 0.0;
    for (int k = 0; k < 3; ++k) {
        double v = fabs(2.0 * sqrt(-Q) * cos((th + 2.0 * k * pi) / 3.0) + 1.0 / 3.0 * I1);
        if (v == v && v > best) best = v;
    }
    return best;
}

__device__ __forceinline__ void atomic_max_nonneg(double* a, double v) {
    atomicMax((unsigned long long*)a, (unsigned long long)__double_as_longlong(v));
}

template <typename T>
__global__ void __launch_bounds__(256) k_monitors(PView<T> P, const uint8_t* __restrict__ mask, double* acc) {
    __shared__ double sh[8][17];
    __shared__ unsigned long long shc[8][5];
    long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long np = P.n;
    double v[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) v[k] = 0.0;
    unsigned long long cnt[5] = {0, 0, 0, 0, 0};
    if (p < np) {
        const unsigned mk = mask[p];
        const double m = (double)P.mass[p];
        double vel[3] = {(double)P.vel[p], (double)P.vel[np + p], (double)P.vel[2 * np + p]};
        if (mk & 1u) {
            for (int c = 0; c < 3; ++c) v[c] = P.pos[c * np + p];
            cnt[0] = 1;
        }
        if (mk & 2u) {
            for (int c = 0; c < 3; ++c) v[3 + c] = vel[c] * m;
            cnt[1] = 1;
        }
        double sg[6], ep[6];
        for (int c = 0; c < 6; ++c) {
            sg[c] = (double)P.stress[c * np + p];
            ep[c] = (double)P.strain[c * np + p];
        }
        if (mk & 4u) {
            v[6] = principal_abs_max(ep);
            v[7] = principal_abs_max(sg);
            cnt[2] = 1;
        }
        if (mk & 8u) {
            for (int c = 0; c < 3; ++c) {
                v[8 + c] = sg[c];
                v[11 + c] = ep[c];
            }
            cnt[3] = 1;
        }
        if (mk & 16u) {
            double sp = sqrt(vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
            v[14] = 0.5 * m * (sp * sp);
            v[15] = P.e_strain[p];
            v[16] = P.e_plastic[p];
            cnt[4] = 1;
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 17; ++k) {
        for (int off = 16; off > 0; off >>= 1) {
            double o = __shfl_down_sync(FULL_MASK, v[k], off);
            v[k] = (k == 6 || k == 7) ? fmax(v[k], o) : v[k] + o;
        }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
        for (int off = 16; off > 0; off >>= 1) cnt[k] += __shfl_down_sync(FULL_MASK, cnt[k], off);
    if (lane == 0) {
        for (int k = 0; k < 17; ++k) sh[w][k] = v[k];
        for (int k = 0; k < 5; ++k) shc[w][k] = cnt[k];
    }
    __syncthreads();
    if (threadIdx.x < 17) {
        const int k = threadIdx.x;
        double s = sh[0][k];
        for (int ww = 1; ww < (int)(blockDim.x >> 5); ++ww) s = (k == 6 || k == 7) ? fmax(s, sh[ww][k]) : s + sh[ww][k];
        if (k == 6 || k == 7)
            atomic_max_nonneg(&acc[k], s);
        else
            atomicAdd(&acc[k], s);
    } else if (threadIdx.x >= 32 && threadIdx.x < 37) {
        const int k = threadIdx.x - 32;
        unsigned long long s = 0;
        for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) s += shc[ww][k];
        atomicAdd((unsigned long long*)&acc[24 + k], s);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_monitor_force(NView<T> nd, double* acc) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nn = nd.nn;
    double f[3] = {0.0, 0.0, 0.0};
    if (i < nn)
        for (int c = 0; c < 3; ++c) f[c] = (double)nd.ftemp[c * nn + i];
    for (int c = 0; c < 3; ++c) {
        for (int off = 16; off > 0; off >>= 1) f[c] += __shfl_down_sync(FULL_MASK, f[c], off);
        if ((threadIdx.x & 31) == 0) atomicAdd(&acc[17 + c], f[c]);
    }
}

// ---------------------------------------------------------------------------
// Return-map network, finishing pass: apply the network's stress increment
// and dR to each queued particle (dR kept non-negative, as the hardening law
// gives), with the plastic strain increment recovered as de - C^-1 dsigma
// (the compliance of …_VonMisesHardening.cpp:64-71), and re-check a hashed
// fraction of the particles against the exact map computed in FP64 on the
// same inputs (cr_increment_wide; the network's error is recorded; then a
// guard replaces implausible results by that exact map, see below;
// the network's result is kept).
// ---------------------------------------------------------------------------
static __global__ void k_sg_finish(PView<float> P, SurrogateQueue q, MatConst M, int contact, double dt, double inv_yield,
                            float recheck, unsigned long long step, const unsigned long long* step_dev,
                            SurrogateAcc* acc, SurrogateGuard gd) {
    if (step_dev) step = *step_dev;
    const unsigned cnt = (unsigned)min((unsigned long long)*q.count, (unsigned long long)q.cap);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&acc->queued, (unsigned long long)cnt);
    const unsigned thr = (unsigned)(recheck * 4294967296.0f);
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < cnt; s += gridDim.x * blockDim.x) {
        const long long p = q.pidx[s];
        const float* qi = q.in + (long long)s * 13;
        const float* qo = q.out + (long long)s * 7;
        float sig[6], e[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            sig[k] = qi[k];
            e[k] = qi[7 + k];
        }
        const float R = qi[6];
        CrOut<float> o;
#pragma unroll
        for (int k = 0; k < 6; ++k) o.dsig[k] = qo[k];
        o.dR = fmaxf(qo[6], 0.0f);
        const float iE = M.finv_E, nE = M.fnu_over_E, iG = M.finv_G;
        o.deps_p[0] = e[0] - (o.dsig[0] * iE - o.dsig[1] * nE - o.dsig[2] * nE);
        o.deps_p[1] = e[1] - (o.dsig[1] * iE - o.dsig[0] * nE - o.dsig[2] * nE);
        o.deps_p[2] = e[2] - (o.dsig[2] * iE - o.dsig[0] * nE - o.dsig[1] * nE);
        o.deps_p[3] = e[3] - o.dsig[3] * iG;
        o.deps_p[4] = e[4] - o.dsig[4] * iG;
        o.deps_p[5] = e[5] - o.dsig[5] * iG;
        // recheck: a hash of (step, particle) below the fraction
        unsigned long long h = (step + 1) * 0x9e3779b97f4a7c15ULL ^ ((unsigned long long)p * 0xbf58476d1ce4e5b9ULL);
        h = (h ^ (h >> 31)) * 0x94d049bb133111ebULL;
        if ((unsigned)(h >> 32) < thr) {
            // the judge: the exact map in FP64 on the same inputs
            CrOut<double> x;
            cr_increment_wide(M, R, sig, e, x);
            double sq = 0.0, mx = 0.0;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const double d = fabs(fps_f2d(o.dsig[k]) - x.dsig[k]) * inv_yield;
                sq += d * d;
                mx = fmax(mx, d);
            }
            atomicAdd(&acc->rechecked, 1ULL);
            atomicAdd(&acc->sq_err, sq / 6.0);
            atomicMax(reinterpret_cast<unsigned long long*>(&acc->max_err), (unsigned long long)__double_as_longlong(mx));
        }
        // the guard: an input outside the training box, or a result that is not the radial return of its trial
        // state (the new stress off the yield surface k0 + R/sqrt 2, a correction dsigma - D de with a
        // hydrostatic part, or a stress or R increment that differs from the radial return evaluated here in
        // FP32; each by more than tol k0), takes the exact map in FP64 instead
        if (gd.tol > 0.0f) {
            bool ok = true;
#pragma unroll
            for (int c = 0; c < 13; ++c) {
                const float xn = qi[c] * gd.in_inv_scale[c];
                ok = ok && xn >= gd.lo[c] && xn <= gd.hi[c];
            }
            float d[6], sn[6];
            trial_increment<float>(M, e, d);
#pragma unroll
            for (int k = 0; k < 6; ++k) sn[k] = sig[k] + o.dsig[k];
            const float a01 = sn[0] - sn[1], a12 = sn[1] - sn[2], a20 = sn[2] - sn[0];
            const float J2 = (a01 * a01 + a12 * a12 + a20 * a20) * (1.0f / 6.0f) + sn[3] * sn[3] + sn[4] * sn[4] +
                             sn[5] * sn[5];
            const float rad = M.fk0 + R * 0.70710678118654752440f;
            const float hyd = ((o.dsig[0] - d[0]) + (o.dsig[1] - d[1]) + (o.dsig[2] - d[2])) * (1.0f / 3.0f);
            const float lim = gd.tol * M.fk0;
            ok = ok && fabsf(sqrtf(J2) - rad) <= lim && fabsf(hyd) <= lim;
            if (ok) {
                // the direction and the hardening: against the FP32 radial return of the same trial state
                CrTrial<float> tr;
                cr_trial<float>(M, R, sig, e, tr);
                CrOut<float> x;
                cr_return<float>(M, R, sig, e, tr, x);
#pragma unroll
                for (int k = 0; k < 6; ++k) ok = ok && fabsf(o.dsig[k] - x.dsig[k]) <= lim;
                ok = ok && fabsf(o.dR - x.dR) <= lim;
            }
            if (!ok) {
                CrOut<double> w;
                cr_increment_wide(M, R, sig, e, w);
                cr_narrow(w, o);
                atomicAdd(&acc->rejected, 1ULL);
            }
        }
        apply_increment<float>(P, p, sig, e, o, q.vol[s], R, true, contact, dt);
    }
}

}  // namespace mpm
