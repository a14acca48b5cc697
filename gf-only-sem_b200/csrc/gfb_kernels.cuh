// gfb_kernels.cuh -- sm_100a kernels of the CG-SEM elastic time loop.
//
// One time step is the element phase followed by the node phase:
//
//   elem_gather_kernel -- for every cell: gather the predicted displacement
//       through ibool, GLL derivative contractions, stress, weighted
//       transposed-derivative divergence (forward/elastic/src/
//       element_cpu.cpp:19-162), point-force injection (forward/share/src/
//       solver.cpp:577-605).  The cell's force contributions are stored cell
//       by cell.  elem_plane_kernel: the same for wavefields in threes.
//   cell_pml_kernel -- per-cell C-PML (FP64, or FP32 where cells disagree):
//       acceleration term and memory update (forward/share/src/
//       pml.cpp:55-216).
//   node_update_kernel, node_pml_kernel -- sum of the contributions of a
//       node's cells in mesh order (no atomics, bit-reproducible run to run),
//       node-form C-PML, Newmark corrector with the diagonal mass and the
//       legacy velocity damping (solver.cpp:52-69, 564-574), then the
//       predictor of the next step (solver.cpp:40-49), so no separate
//       predictor launch is needed.
//
// elem_col_kernel and elem_pipe_kernel assemble in the element phase instead,
// one launch per colour with a plain read-modify-write of the global force:
// cells of one colour share no node and colours run in a fixed order, and the
// first colour touching a node stores instead of adding, which replaces the
// memset of the global residual (cuda_step.cu:289-290).
//
// Layouts on the device (cells in mesh order):
//   ibool  [cell][NN]            node id | FIRST_TOUCH, LAST_TOUCH bits (by colour)
//   geom   [cell][geo_row] Real  dxi_dx (9), lambda and mu times the weight
//   state  u, v (double), a (Real): [node][3*n_field];
//          predicted displacement ut and force (Real): [node][n_field][4]
//   C-PML  coef [slot][15][NN] Real (alpha 9, abar 5, w*J/rho),
//          mem [slot][n_field*9][NN], prev [slot][n_field*3][NN]
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gfb {

constexpr uint32_t kFirstTouch = 0x80000000u;  // lowest colour touching the node: store
constexpr uint32_t kLastTouch = 0x40000000u;   // highest colour touching the node: finalise
constexpr uint32_t kNodeMask = 0x3fffffffu;

// Predicted displacement and force of the time loop are stored
// [node][field][4] (x, y, z, pad) so a field of a node is one 16-byte
// vector; u, v, a are [node][3*field].  Index of component f of node g.
__device__ __forceinline__ long long padded_index(long long g, int f, int F) {
    return g * (F / 3) * 4 + (f / 3) * 4 + (f % 3);
}

// Node-table rows used by the pipelined kernels: the NN node words of a
// cell, then the index of the model the cell belongs to, padded to whole
// 16-byte copies.
__host__ __device__ constexpr int ib_row_words(int nn) { return (nn + 1 + 3) / 4 * 4; }

// Geometry rows of the time loop, [cell][geo_row]: dxi_dx (9 x NN), then
// lambda and mu times det J w_i w_j w_k (so the stress they give is already
// the flux's and the weight costs no load or multiply), padded to whole
// 16-byte copies.  Where mu <= 0 both are 0: the point adds nothing, whatever
// its other values are (element_cpu.cpp:42-43).
template <typename Real>
__host__ __device__ constexpr int geo_row(int nn) {
    return (11 * nn * (int)sizeof(Real) + 15) / 16 * 16 / (int)sizeof(Real);
}

// Time-step constants of one model (several independent models can share
// one solver): dt, dt^2/2 (beta = 0) and the C-PML field coefficients
// c1 = (1-2 theta) dt/2, c2 = (1-theta) dt^2/2 of pml.cpp:35, 63-64.
struct ModelConst {
    double dt, half_dt2, c1, c2;
};
constexpr int kMaxModels = 255;
// Wavefields one solver advances together: force directions times source
// positions (a source set per position, each with its cells, weights and
// source time function).
constexpr int kMaxFields = 12;

// Direction and source set of wavefield f (kernel parameters are indexed
// with compile-time indices only).
template <int NFLD>
__device__ __forceinline__ void field_source(const int (&dir)[kMaxFields], const int (&fset)[kMaxFields], int f,
                                             int& d, int& k) {
    d = dir[0];
    k = fset[0];
#pragma unroll
    for (int q = 1; q < NFLD; ++q)
        if (f == q) {
            d = dir[q];
            k = fset[q];
        }
}

template <int NG>
struct Shape {
    static constexpr int NN = NG * NG * NG;
    static constexpr int NNP = (NN + 31) / 32 * 32;
};

// Assembly by the node pass.  The element kernel leaves every cell's force
// contributions in contrib [cell][chunk][NN][fields of the chunk][3], cells in
// mesh order: a chunk holds up to gather_chunk_fields wavefields, so what a
// node reads of a cell is contiguous, as its state is.  A touch is an index
// into it in units of 3 Reals (of the point's first wavefield, chunk 0); a
// node's touches in mesh order:
//   touch[g].x .y .z  the first three (kNoTouch: fewer)
//   touch[g].w        the fourth, kNoTouch, or kMoreTouches | i: the touches
//                     from the fourth on are more[i] (and more[i+1], ... while
//                     bit 31 of .x is set), unused entries kNoTouch.
// All but the corner nodes of a hexahedral mesh (1 in 64 at ngll 5) have at
// most four touches and need this one 16-byte entry.  The sum runs in mesh
// order.
constexpr uint32_t kNoTouch = 0xffffffffu;
constexpr uint32_t kMoreTouches = 0x80000000u;
template <typename Real>
__host__ __device__ constexpr int gather_chunk_fields(int nfld) {
    return sizeof(Real) == 8 ? 1 : (nfld < 3 ? nfld : 3);
}
// Units (3 Reals) of a chunk: whole 16-byte copies.
template <typename Real>
__host__ __device__ constexpr int gather_chunk_units(int nn, int nfld) {
    return (nn * gather_chunk_fields<Real>(nfld) * 3 * (int)sizeof(Real) + 47) / 48 * 48 / (3 * (int)sizeof(Real));
}
template <typename Real>
struct NodeGather {
    const uint4* touch;
    const uint4* more;
    const Real* contrib;
    int chunk_units;
    bool keep;              // the assembled force is kept in `force` (increments, records)
    const int* mdirect;     // [model] 0: this step's contributions add to the kept force (nullptr: in full)
};

template <typename Real>
struct NodeArgs {
    long long n_node;
    double* u;              // [node][3*n_field]
    double* v;
    Real* a;
    Real* ut;               // [node][field][4]
    Real* force;            // [node][field][4]
    NodeGather<Real> gather;  // cell contributions to assemble (touch == nullptr: `force` is assembled)
    const double* mass;     // [n_node] assembled lumped mass
    const Real* inv_mass;   // [n_node] 1/m (FP32 path) or nullptr
    const double* damping;  // [n_node] or nullptr
    double dt, half_dt2, beta, gamma;
    // several models: model of each node, its constants, whether it still steps
    const uint8_t* node_model;
    const ModelConst* mc;
    const int* mlive;
    const long long* live_node_end;  // [2] end of the stepping C-PML / plain nodes (several models), or null
    // [model] 1 when the model's next step evaluates the element force in
    // full (the node pass then stores the predicted displacement), 0 when
    // it adds the force of the step's increment (the node pass stores the
    // increment of the predicted displacement); nullptr: always in full
    const int* mnext;
    // plain nodes keep the half-step velocity w = v + dt/2 a (in float, in
    // w32 [node][3*n_field]) and no acceleration (see update_node_field)
    bool half_v;
    float* w32;
};

// C-PML at global nodes (FP32 path).
//
// The reference keeps C-PML memory per cell and GLL node (pml.cpp:112-149)
// and adds each cell's term w J/rho (A1 v + A2 u + A3 m_x + A4 m_y + A5 m_z)
// to the cell residual before assembly (pml.cpp:151-216).  At a node shared
// by several C-PML cells the memory of an axis that is active in those
// cells follows the same recursion m = a0 m + a1 new + a2 old with the same
// new/old (they are node values) and the same axis coefficients (functions
// of the node position), and A_{3+q} = 0 exactly in cells where axis q is
// inactive.  So the memory is kept once per node and axis, and the assembled
// term is B1 v + B2 u + B3 m_x + B4 m_y + B5 m_z with B_k = sum over the
// node's C-PML cells of w J/rho A_k.  The host checks the axis coefficients
// agree across cells before choosing this form.
// The C-PML nodes are the device nodes [0, n_slot): a node's slot is its
// index.
template <typename Real>
struct NodePml {
    const Real* coef;    // [slot][14]: B1..B5, alpha x(3), y(3), z(3)
    Real* mem;           // [axis][slot][F]; only live axes are read or written
    Real* prev;          // [slot][F]  last step's u + c1 v
    long long n_slot;
    double c1, c2;
};

template <typename Real>
struct ElemArgs {
    int e_begin, e_end;     // range of `cells`
    const int* cells;       // the cells colour after colour
    const Real* geom;
    const Real* ut;
    Real* force;
    const Real* dmat;  // [NG*NG]
    // C-PML
    const int* pml_slot;   // [cell] -1 if not a C-PML cell
    const Real* pml_coef;  // [slot][15][NN]
    Real* pml_mem;         // [slot][F*3][NN]
    Real* pml_prev;        // [slot][F][NN]
    const double* u;     // [node][3*n_field]
    const double* v;
    const Real* a;
    long long n_node;
    double c1, c2;
    // source
    const int* src_head;  // [cell] first source slot or -1
    const int* src_next;  // [slot]
    const Real* src_w;    // [slot][NN]
    const Real* mstf;     // [model][set] source time function value of this step (nullptr: none)
    const int* src_set;   // [slot] source set of the slot (nullptr: every slot is set 0)
    int n_set;            // source sets (one per source position)
    const int* mlive;     // [model] 1 while the model still steps
    const int* mdirect;   // [model] 1: this step evaluates the force in full (first touch stores), 0: adds the
                          // increment's force to the stored one; nullptr: in full
    const ModelConst* mc; // [model]
    int dir[kMaxFields];  // force direction of each wavefield
    int fset[kMaxFields]; // source set of each wavefield
    // finalisation of the nodes whose last touching colour this is (the
    // node update fused into the element kernel); fuse == 0 keeps the
    // force in memory for a separate node pass
    int fuse;
    NodeArgs<Real> nu;
    NodePml<Real> np;
};

// 16-byte vector helpers (a float4, or two double2 for FP64 vectors).
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(double* p, double a, double b, double c, double d) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
    reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// FP64 operations rounded one by one (no contraction into FMA), so that the
// node update rounds the same way in every instantiation of the kernels
// that inline it (a solver of one model and of several must agree bit for
// bit) and in the reference's evaluation order.
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }

// Programmatic dependent launch along a step: step start -> element kernel ->
// node passes -> next step's start.  A kernel launched this way may start
// before the one before it has finished: it sets itself up from arrays no
// kernel writes (node words, geometry, touches, C-PML coefficients), then
// pdl_wait() returns when the kernels that it depends on directly (both node
// passes: the element kernel; the next step's start: both node passes) have
// completed and their writes, and what those were ordered after, are visible.
// Every thread reads and writes what a kernel of the chain writes only after
// its own pdl_wait(), and every kernel calls it before it ends, so its
// completion implies that of all before it.  pdl_launch(): the next kernel may
// start now; it comes after pdl_wait(), so no kernel starts before the ones
// two before it have completed.  What a kernel of the chain writes is read with
// ordinary or L2 loads, not through the read-only path.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Real operations rounded the same way wherever the node update is inlined
// (node passes, fused update).
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }

// One wavefield of a node on its way through the end of a step: load() issues
// every load, finish() takes the complete assembled force fv through the node
// C-PML term (when PML and pml), the Newmark corrector with the diagonal mass
// (solver.cpp:52-69, legacy damping of 564-574 applied to v first) and the
// next step's predictor (40-49).  On the FP32 path 1/m == 0 marks a node with
// m <= 0 (the host stores 0 there), so the f64 mass is not read.
// HALF_V: Newmark with beta = 0, gamma = 1/2 (solver.cpp:40-69) written on
// the half-step velocity w = v + dt/2 a: u_{n+1} = u_n + dt w_n, a_{n+1} = f/m,
// w_{n+1} = w_n + dt a_{n+1}, and the next predicted displacement
// u_{n+1} + dt w_{n+1} (its increment dt w_{n+1}).  The same values as the
// (u, v, a) form in exact arithmetic, without the acceleration's read and
// write; v and a are recovered from w and the assembled force when they are
// needed (records, state).  w is held in float (its rounding adds a random
// walk of ~1e-7 relative per step, far below the float rounding of the
// predicted displacement that bounds this path), u in double.
template <typename Real, int NFLD, bool PML, bool HALF_V>
struct NodeField {
    static constexpr int F = 3 * NFLD;
    double u[3], v[3], m, dmp;
    Real a[3], im;
    float w[3];
    Real mm[3][3], pr[3];

    // cf: the node's C-PML coefficients (when pml)
    __device__ __forceinline__ void load(const NodeArgs<Real>& A, const NodePml<Real>& P, long long g, int d, bool pml,
                                         const Real* cf) {
        const size_t i = (size_t)g * F + d * 3;
        im = A.inv_mass ? __ldg(A.inv_mass + g) : Real(0);
#pragma unroll
        for (int c = 0; c < 3; ++c) u[c] = A.u[i + c];
        if constexpr (HALF_V) {
#pragma unroll
            for (int c = 0; c < 3; ++c) w[c] = A.w32[i + c];
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[c] = A.v[i + c];
                a[c] = A.a[i + c];
            }
            m = A.inv_mass ? 1.0 : __ldg(A.mass + g);
            dmp = A.damping ? __ldg(A.damping + g) : 0.0;
            if (PML && pml) {
#pragma unroll
                for (int c = 0; c < 3; ++c) pr[c] = P.prev[i + c];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const Real* mem = P.mem + (size_t)q * P.n_slot * F + i;
                    const bool live = cf[2 + q] != Real(0);
#pragma unroll
                    for (int c = 0; c < 3; ++c) mm[q][c] = live ? mem[c] : Real(0);
                }
            }
        }
    }

    __device__ __forceinline__ void finish(const NodeArgs<Real>& A, const NodePml<Real>& P, long long g, int d, bool pml,
                                           const Real* cf, const Real (&fv)[3], const ModelConst& K, bool full) {
        const size_t i = (size_t)g * F + d * 3;
        Real out[3];
        if constexpr (HALF_V) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double ww = (double)w[c];
                if (im != Real(0)) {  // m <= 0: the node stays as it is (a = 0, solver.cpp:58-61)
                    const double a_new = (double)rmul(fv[c], im);
                    u[c] = dadd(u[c], dmul(K.dt, ww));
                    ww = (double)(float)dadd(ww, dmul(K.dt, a_new));
                    A.u[i + c] = u[c];
                    A.w32[i + c] = (float)ww;
                }
                out[c] = full ? (Real)dadd(u[c], dmul(K.dt, ww)) : (Real)dmul(K.dt, ww);
            }
        } else {
            const bool massless = A.inv_mass ? (im == Real(0)) : (m <= 0.0);
            Real force[3] = {fv[0], fv[1], fv[2]};
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (dmp > 0.0) v[c] = __dsub_rn(v[c], dmul(dmp, v[c]));
            if (PML && pml) {
                Real nv[3], ov[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    nv[c] = (Real)dadd(u[c], dmul(K.c1, v[c]));
                    ov[c] = rfma((Real)K.c2, a[c], pr[c]);
                    Real t = rmul(cf[0], (Real)v[c]);
                    t = rfma(cf[1], (Real)u[c], t);
#pragma unroll
                    for (int q = 0; q < 3; ++q) t = rfma(cf[2 + q], mm[q][c], t);
                    force[c] += t;
                    P.prev[i + c] = nv[c];
                }
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (cf[2 + q] != Real(0)) {
                        Real* mem = P.mem + (size_t)q * P.n_slot * F + i;
                        const Real k0 = cf[5 + 3 * q], k1 = cf[6 + 3 * q], k2 = cf[7 + 3 * q];
#pragma unroll
                        for (int c = 0; c < 3; ++c) mem[c] = rfma(k2, ov[c], rfma(k1, nv[c], rmul(k0, mm[q][c])));
                    }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double a_new = 0.0;
                if (!massless) {
                    a_new = A.inv_mass ? (double)rmul(force[c], im) : __ddiv_rn((double)force[c], m);
                    a_new = (double)(Real)a_new;
                    const double a_old = (double)a[c];
                    // solver.cpp:62-66
                    const double ta = dadd(dmul(0.5 - A.beta, a_old), dmul(A.beta, a_new));
                    u[c] = dadd(u[c], dadd(dmul(K.dt, v[c]), dmul(dmul(K.dt, K.dt), ta)));
                    v[c] = dadd(v[c], dmul(K.dt, dadd(dmul(1.0 - A.gamma, a_old), dmul(A.gamma, a_new))));
                }
                A.u[i + c] = u[c];
                A.v[i + c] = v[c];
                A.a[i + c] = (Real)a_new;
                // the next step's predicted displacement (solver.cpp:40-49), or its
                // increment over this step's (u_{n+1} is this step's prediction)
                const double inc = dadd(dmul(K.dt, v[c]), dmul(K.half_dt2, a_new));
                out[c] = full ? (Real)dadd(u[c], inc) : (Real)inc;
            }
        }
        store4(A.ut + ((size_t)g * NFLD + d) * 4, out[0], out[1], out[2], Real(0));
    }
};

// Wavefield d of node g finalised from its complete assembled force (the
// node update fused into the element kernel).
template <typename Real, int NFLD, bool PML>
__device__ __forceinline__ void update_node_field(const NodeArgs<Real>& A, const NodePml<Real>& P, long long g,
                                                  int d, const Real (&fv)[3], int sl, const ModelConst& K,
                                                  bool full = true) {
    NodeField<Real, NFLD, PML, false> x;
    Real cf[14];
    if (PML && sl >= 0) {
#pragma unroll
        for (int q = 0; q < 14; ++q) cf[q] = __ldg(P.coef + (size_t)sl * 14 + q);
    }
    x.load(A, P, g, d, sl >= 0, cf);
    x.finish(A, P, g, d, sl >= 0, cf, fv, K, full);
}

// Constants of the model node g belongs to; false when that model has
// taken all its steps (its state stays as it is).
template <typename Real, bool MULTI>
__device__ __forceinline__ bool node_constants(const NodeArgs<Real>& A, const NodePml<Real>& P, long long g,
                                               ModelConst& K, bool& full) {
    if (!MULTI) {
        K = ModelConst{A.dt, A.half_dt2, P.c1, P.c2};
        full = A.mnext ? A.mnext[0] != 0 : true;
        return true;
    }
    const int m = __ldg(A.node_model + g);
    if (!__ldcg(A.mlive + m)) return false;
    K = A.mc[m];
    full = A.mnext ? A.mnext[m] != 0 : true;
    return true;
}

// The parts of the assembled force of a node's wavefield, loaded: the kept
// force (add: the contributions add to it) and the first four touches.
template <typename Real, int NFLD>
struct ForceParts {
    Real old[4], c[4][3];
    static __device__ __forceinline__ const Real* touches(const NodeArgs<Real>& A, int d) {
        constexpr int FC = gather_chunk_fields<Real>(NFLD);
        return A.gather.contrib + ((size_t)(d / FC) * A.gather.chunk_units + d % FC) * 3;
    }
    static __device__ __forceinline__ void touch(const Real* base, uint32_t q, bool on, Real (&x)[3]) {
        const Real* p = base + (size_t)q * 3;
#pragma unroll
        for (int k = 0; k < 3; ++k) x[k] = on ? p[k] : Real(0);
    }
    __device__ __forceinline__ void load(const NodeArgs<Real>& A, long long g, int d, const uint4& t, bool add) {
        const Real* base = touches(A, d);
        touch(base, t.x, t.x != kNoTouch, c[0]);
        touch(base, t.y, t.y != kNoTouch, c[1]);
        touch(base, t.z, t.z != kNoTouch, c[2]);
        touch(base, t.w, !(t.w & kMoreTouches), c[3]);
        old[0] = old[1] = old[2] = Real(0);
        if (add) load4(A.force + ((size_t)g * NFLD + d) * 4, old);
    }
    __device__ __forceinline__ void sum(const NodeArgs<Real>& A, int d, const uint4& t, Real (&fv)[3]) const {
        Real s[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s[k] = c[0][k] + c[1][k];
            s[k] += c[2][k];
            s[k] += c[3][k];
        }
        if ((t.w & kMoreTouches) && t.w != kNoTouch) {
            const Real* base = touches(A, d);
            const uint4* m = A.gather.more + (t.w & ~kMoreTouches);
            bool on = true;
            while (on) {
                const uint4 q = __ldg(m++);
                on = (q.x & kMoreTouches) != 0;
                Real x[4][3];
                touch(base, q.x & ~kMoreTouches, true, x[0]);
                touch(base, q.y, q.y != kNoTouch, x[1]);
                touch(base, q.z, q.z != kNoTouch, x[2]);
                touch(base, q.w, q.w != kNoTouch, x[3]);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    s[k] += x[0][k];
                    s[k] += x[1][k];
                    s[k] += x[2][k];
                    s[k] += x[3][k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) fv[k] = old[k] + s[k];
    }
};

// Node pass: one thread per (node, wavefield), the wavefields of a node in
// adjacent threads, so a warp reads and writes whole rows of u, v, a and of a
// cell's contributions.  A warp takes 32 nodes at a time, every load of a
// thread issued before its first store; their touches and C-PML coefficients,
// which the other addresses wait for, come through the warp's own shared memory
// two tiles ahead (cp.async), so the warps run without block barriers.  With node-form C-PML the pass is
// two launches over contiguous node ranges, side by side on two streams:
// node_update_kernel over the plain nodes [g0, n_node), node_pml_kernel over the
// C-PML nodes [0, g0).
constexpr int kNodeThreads = 128, kNodeTile = 32;

template <typename Real, int NFLD, bool MULTI, bool PML, bool HALF_V>
__device__ __forceinline__ void node_pass(const NodeArgs<Real>& A, const NodePml<Real>& P, long long g0) {
    constexpr int TN = kNodeTile, WARPS = kNodeThreads / 32;
    constexpr int COEF_W = 16 / (int)sizeof(Real), COEF_N = PML ? TN * 14 : COEF_W;
    __shared__ __align__(16) uint4 s_touch[WARPS][3][TN];
    __shared__ __align__(16) Real s_cf[PML ? WARPS : 1][3][COEF_N];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const bool gather = A.gather.touch != nullptr;
    long long g1 = PML ? P.n_slot : A.n_node;
    if (MULTI && A.live_node_end) {  // this step's bounds
        pdl_wait();
        g1 = min(g1, A.live_node_end[PML ? 0 : 1]);
    }
    const long long n_tile = (g1 - g0 + TN - 1) / TN;
    const long long step = (long long)gridDim.x * WARPS;
    auto fetch = [&](long long tile, int st) {
        if (tile < n_tile) {
            const long long b = g0 + tile * TN;
            const int n = (int)min((long long)TN, g1 - b);
            if (gather && lane < n) cp_async16(&s_touch[wp][st][lane], A.gather.touch + b + lane);
            if (PML)  // the coefficient array is padded to whole copies
                for (int i = lane; i * COEF_W < n * 14; i += 32)
                    cp_async16(&s_cf[PML ? wp : 0][st][i * COEF_W], P.coef + b * 14 + i * COEF_W);
        }
        cp_async_commit();
    };
    const long long first = (long long)blockIdx.x * WARPS + wp;
    fetch(first, 0);
    fetch(first + step, 1);
    pdl_wait();
    pdl_launch();
    ModelConst K;
    bool full, add = false;
    if (!MULTI) {
        node_constants<Real, MULTI>(A, P, 0, K, full);
        add = A.gather.keep && A.gather.mdirect && __ldcg(A.gather.mdirect) == 0;
    }
    int st = 0;
    for (long long tile = first; tile < n_tile; tile += step) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();  // this tile's tables; and every lane is done with the tile before
        fetch(tile + 2 * step, st >= 1 ? st - 1 : 2);
        const long long b = g0 + tile * TN;
        const int n = (int)min((long long)TN, g1 - b) * NFLD;
#pragma unroll 1
        for (int r = 0; r < NFLD; ++r) {
            const int s = r * 32 + lane;
            if (s >= n) continue;
            const int gl = s / NFLD, d = s - gl * NFLD;
            const long long g = b + gl;
            if (MULTI && !node_constants<Real, MULTI>(A, P, g, K, full)) continue;
            const uint4 t = s_touch[wp][st][gl];
            const Real* cf = &s_cf[PML ? wp : 0][st][PML ? gl * 14 : 0];
            NodeField<Real, NFLD, PML, HALF_V> x;
            ForceParts<Real, NFLD> p;
            if (gather) {
                if (MULTI)
                    add = A.gather.keep && A.gather.mdirect && __ldcg(A.gather.mdirect + __ldg(A.node_model + g)) == 0;
                p.load(A, g, d, t, add);
            } else {
                load4(A.force + ((size_t)g * NFLD + d) * 4, p.old);
            }
            x.load(A, P, g, d, true, cf);
            Real fv[3] = {p.old[0], p.old[1], p.old[2]};
            if (gather) p.sum(A, d, t, fv);
            x.finish(A, P, g, d, true, cf, fv, K, full);
            if (A.gather.keep) store4(A.force + ((size_t)g * NFLD + d) * 4, fv[0], fv[1], fv[2], Real(0));
        }
        st = st == 2 ? 0 : st + 1;
    }
    cp_async_wait_all();
}

// Resident blocks per SM.  The passes are bound by DRAM and by the loads in
// flight: on 40 x 40 x 20 cells (1.06 M plain and 1.03 M C-PML nodes, three
// wavefields) the plain pass takes 102 / 89 / 120 us with 6 / 8 / 10 blocks
// (72 / 64 / 48 registers, the last with spills), the C-PML pass 157 / 146 /
// 200 us with 5 / 6 / 8 (96 / 80 / 64), 5.3 and 5.5 TB/s of DRAM traffic at
// the best.  Three wavefields per thread at once (128 registers) or whole
// tiles by bulk copies (fewer warps, by shared memory) were slower.
template <typename Real>
constexpr int node_blocks_per_sm(bool pml) {
    return pml ? 6 : (sizeof(Real) == 4 ? 8 : 5);
}

template <typename Real, int NFLD, bool MULTI, bool HALF_V>
__global__ void __launch_bounds__(kNodeThreads, node_blocks_per_sm<Real>(false))
    node_update_kernel(const __grid_constant__ NodeArgs<Real> A, const __grid_constant__ NodePml<Real> P, long long g0) {
    node_pass<Real, NFLD, MULTI, false, HALF_V>(A, P, g0);
}

template <int NFLD, bool MULTI>
__global__ void __launch_bounds__(kNodeThreads, node_blocks_per_sm<float>(true))
    node_pml_kernel(const __grid_constant__ NodeArgs<float> A, const __grid_constant__ NodePml<float> P) {
    node_pass<float, NFLD, MULTI, true, false>(A, P, 0);
}

// The assembled force alone (a learned layer adds to it between the element
// and the node phase; the autotuner times it).
template <typename Real, int NFLD, bool MULTI>
__global__ void __launch_bounds__(256) assemble_kernel(NodeArgs<Real> A, NodePml<Real> P) {
    const long long total = A.n_node * NFLD;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
        const long long g = t / NFLD;
        const int d = (int)(t - g * NFLD);
        ModelConst K;
        bool full;
        if (!node_constants<Real, MULTI>(A, P, g, K, full)) continue;
        const uint4 q = __ldg(A.gather.touch + g);
        ForceParts<Real, NFLD> p;
        p.load(A, g, d, q, A.gather.keep && A.gather.mdirect && __ldg(A.gather.mdirect + (MULTI ? __ldg(A.node_model + g) : 0)) == 0);
        Real fv[3];
        p.sum(A, d, q, fv);
        store4(A.force + ((size_t)g * NFLD + d) * 4, fv[0], fv[1], fv[2], Real(0));
    }
}

// Start of a step for every model: whether it still steps, and its source
// time function value (solver.cpp:577-605 uses stf_values[step]; steps past
// the end of the series inject nothing).  mstep[m] is the step about to be
// computed and moves on by one while the model steps, so a captured step
// replays correctly.
// Series q = m * n_set + k is source set k of model m.
//
// Element force in full or by increments: a step whose element phase
// evaluates the force of the full predicted displacement (mdirect = 1: the
// first colour touching a node stores) is followed by up to period-1 steps
// that add the force of the predicted displacement's increment to the
// stored force (mdirect = 0); the source then adds the increment of the
// source time function.  A one-shot force_direct[m] (set by the host after
// the predicted displacement was rewritten from u, v, a) makes the step a
// full one.  mnext[m] tells the node pass what the next step needs.
template <typename Real>
__global__ void step_begin_kernel(int n_model, int n_set, int* mstep, const int* nsteps, const int* n_stf,
                                  const long long* stf_off, const Real* stf_all, Real* mstf, int* mlive, int period,
                                  int* force_direct, int* mdirect, int* mnext) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    pdl_launch();
    if (m >= n_model) return;
    const int t = mstep[m];
    const bool live = t < nsteps[m];
    mlive[m] = live ? 1 : 0;
    bool full = true;
    if (mdirect) {
        full = period <= 1 || force_direct[m] != 0 || t % period == 0;
        force_direct[m] = 0;
        mdirect[m] = full ? 1 : 0;
        mnext[m] = (period <= 1 || (t + 1) % period == 0) ? 1 : 0;
    }
    for (int k = 0; k < n_set; ++k) {
        const int q = m * n_set + k;
        const Real now = (live && t < n_stf[q]) ? stf_all[stf_off[q] + t] : Real(0);
        const Real before = (!full && t >= 1 && t - 1 < n_stf[q]) ? stf_all[stf_off[q] + t - 1] : Real(0);
        mstf[q] = full ? now : (live ? now - before : Real(0));
    }
    mstep[m] = t + (live ? 1 : 0);
}

// Several models in one solver: after step_begin_kernel, the end of the
// cells still stepping in each colour and of the nodes still stepping in the
// C-PML and plain node ranges.  Cells of a colour and nodes of a range are
// grouped by model, so everything past the largest end of a live model
// belongs to finished models and the launches of this step stop there
// (cells and nodes before it of finished models are still skipped one by
// one).  cell_end [model][colour], node_end [model][2] (C-PML, plain); one
// block, a thread per colour or range.
static __global__ void live_bounds_kernel(int n_model, int n_colour, const int* mlive, const int* cell_end,
                                   const int* colour_first, const long long* node_end, long long plain_first,
                                   int* live_cell_end, long long* live_node_end) {
    pdl_wait();
    pdl_launch();
    for (int c = threadIdx.x; c < n_colour + 2; c += blockDim.x) {
        if (c < n_colour) {
            int e = colour_first[c];
            for (int m = 0; m < n_model; ++m)
                if (mlive[m]) e = max(e, cell_end[m * n_colour + c]);
            live_cell_end[c] = e;
        } else {
            const int r = c - n_colour;
            long long g = r == 0 ? 0 : plain_first;
            for (int m = 0; m < n_model; ++m)
                if (mlive[m]) g = max(g, node_end[m * 2 + r]);
            live_node_end[r] = g;
        }
    }
}

// ---------------------------------------------------------------------------
// elem_pipe_kernel: persistent, software-pipelined element/assembly kernel.
//
// Blocks loop over groups of EPB cells of one colour.  While group i is
// computed, the gathered displacement of group i+1 and the geometry + node
// table of group i+2 are in flight as cp.async copies into rotating shared
// stages (3 stages for geometry/ibool, 2 for the gathered vectors), so each
// SM keeps tens of KB of loads outstanding independent of how many blocks
// fit.  Thread per GLL point; the n_field wavefields are looped per thread.
// Node table rows on the device hold the cell's model index after its node
// words and are padded so every copy is a 16-byte cp.async.
// ---------------------------------------------------------------------------

// Bulk copies (TMA, no tensor map, no multicast) completing on an mbarrier
// of this block: one thread announces the bytes of a stage and issues its
// copies; every thread waits for the phase with a bounded poll.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// The phase of parity `parity` completed; false after kMbarPolls polls
// (each try_wait may suspend the thread for a while), which only a lost
// copy would cause.
constexpr long kMbarPolls = 1L << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    for (long k = 0; k < kMbarPolls; ++k)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
// bytes: a multiple of 16; both addresses 16-byte aligned
__device__ __forceinline__ void bulk_copy_g2s(void* smem, const void* gmem, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// A chunk of shared memory to global memory, in the issuing thread's current
// bulk group; bulk_wait_read: the groups committed so far have read their
// shared memory, bulk_wait_all: and written their global memory.
__device__ __forceinline__ void bulk_copy_s2g(void* gmem, const void* smem, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gmem), "r"(smem_u32(smem)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

template <typename Real, int NG, int NFLD>
struct PipeShape {
    static constexpr int NN = NG * NG * NG;
    static constexpr int NNP = (NN + 31) / 32 * 32;
    static constexpr int EPB = NNP <= 32 ? 8 : (NNP <= 64 ? 4 : (NNP <= 128 ? 2 : 1));
    static constexpr int THREADS = NNP * EPB;
    static constexpr int GEO_B = geo_row<Real>(NN) * (int)sizeof(Real); // geometry bytes per cell
    static constexpr int IB_B = ib_row_words(NN) * 4;                  // node-table bytes per cell
    static constexpr int BUF_B = NN * NFLD * 4 * (int)sizeof(Real);    // field vectors per cell
    // a geometry stage also receives the cell's old force vectors once the
    // geometry has been read into registers
    static constexpr int GEO_SLOT = GEO_B > BUF_B ? GEO_B : BUF_B;
    static constexpr int GSTAGE = EPB * GEO_SLOT;
    static constexpr int ISTAGE = EPB * IB_B;
    static constexpr int BSTAGE = EPB * BUF_B;
    static constexpr int D_B = 64 * (int)sizeof(Real);
    static constexpr int SMEM = D_B + 2 * GSTAGE + 3 * ISTAGE + 2 * BSTAGE;
    static constexpr int MIN_BLOCKS = (64 * 1024) / (THREADS * 64) > 0 ? (64 * 1024) / (THREADS * 64) : 1;
    static_assert(GEO_B % 16 == 0 && IB_B % 16 == 0 && BUF_B % 16 == 0, "16-byte copies");
};

template <typename Real, int NG, int NFLD>
__global__ void __launch_bounds__(PipeShape<Real, NG, NFLD>::THREADS, (sizeof(Real) == 4 ? PipeShape<Real, NG, NFLD>::MIN_BLOCKS : 1))
    elem_pipe_kernel(ElemArgs<Real> A, const uint32_t* __restrict__ ibool_padded, int n_groups) {
    using S = PipeShape<Real, NG, NFLD>;
    constexpr int NN = S::NN, NNP = S::NNP, EPB = S::EPB, THREADS = S::THREADS;
    constexpr int VW = 16 / (int)sizeof(Real);               // Reals per 16-byte copy
    constexpr int CPV = 4 * (int)sizeof(Real) / 16;          // 16-byte copies per field vector
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real* sD = reinterpret_cast<Real*>(smem_raw);
    unsigned char* gbase = smem_raw + S::D_B;
    unsigned char* ibase = gbase + 2 * S::GSTAGE;
    unsigned char* bbase = ibase + 3 * S::ISTAGE;
    const int tid = threadIdx.x;
    const int el = tid / NNP, p = tid - el * NNP;
    if (tid < NG * NG) sD[tid] = A.dmat[tid];

    auto geo_of = [&](int st, int c) -> Real* {
        return reinterpret_cast<Real*>(gbase + st * S::GSTAGE + c * S::GEO_SLOT);
    };
    auto ib_of = [&](int st, int c) -> uint32_t* {
        return reinterpret_cast<uint32_t*>(ibase + st * S::ISTAGE + c * S::IB_B);
    };
    auto buf_of = [&](int st, int c) -> Real* {
        return reinterpret_cast<Real*>(bbase + st * S::BSTAGE + c * S::BUF_B);
    };
    auto issue_ib = [&](int grp, int st) {
        constexpr int CI = S::IB_B / 16;
        for (int q = tid; q < EPB * CI; q += THREADS) {
            const int c = q / CI, r = q - c * CI;
            const int x = A.e_begin + grp * EPB + c;
            if (x < A.e_end)
                cp_async16(reinterpret_cast<unsigned char*>(ib_of(st, c)) + r * 16,
                           reinterpret_cast<const unsigned char*>(ibool_padded) + (size_t)__ldg(A.cells + x) * S::IB_B + r * 16);
        }
    };
    auto issue_geo = [&](int grp, int st) {
        constexpr int CG = S::GEO_B / 16;
        for (int q = tid; q < EPB * CG; q += THREADS) {
            const int c = q / CG, r = q - c * CG;
            const int x = A.e_begin + grp * EPB + c;
            if (x < A.e_end)
                cp_async16(reinterpret_cast<unsigned char*>(geo_of(st, c)) + r * 16,
                           reinterpret_cast<const unsigned char*>(A.geom) + (size_t)__ldg(A.cells + x) * S::GEO_B + r * 16);
        }
    };
    // this point's predicted-displacement vectors (node table in stage ist)
    auto issue_gather = [&](int grp, int ist, int bs) {
        if (A.e_begin + grp * EPB + el >= A.e_end || p >= NN) return;
        const uint32_t g = ib_of(ist, el)[p] & kNodeMask;
#pragma unroll
        for (int d = 0; d < NFLD; ++d)
#pragma unroll
            for (int h = 0; h < CPV; ++h)
                cp_async16(buf_of(bs, el) + (p * NFLD + d) * 4 + h * VW, A.ut + ((size_t)g * NFLD + d) * 4 + h * VW);
    };

    // prologue: node table of the first group, then its vectors and
    // geometry and the node table of the second group
    const int grp0 = blockIdx.x;
    if (grp0 < n_groups) issue_ib(grp0, 0);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (grp0 < n_groups) {
        issue_gather(grp0, 0, 0);
        issue_geo(grp0, 0);
    }
    if (grp0 + (int)gridDim.x < n_groups) issue_ib(grp0 + gridDim.x, 1);
    cp_async_commit();

    const int i = p / (NG * NG), j = (p / NG) % NG, k = p % NG;
    int it = 0;
    for (int grp = grp0; grp < n_groups; grp += gridDim.x, ++it) {
        const int cur = it & 1, ist = it % 3;
        cp_async_wait_all();
        __syncthreads();  // vectors + geometry of this group, node table of the next
        const bool in = A.e_begin + grp * EPB + el < A.e_end;
        const int e = in ? __ldg(A.cells + A.e_begin + grp * EPB + el) : 0;
        const int mdl = in ? (int)ib_of(ist, el)[NN] : 0;
        const bool active = in && (p < NN) && (!A.mlive || __ldg(A.mlive + mdl));
        const uint32_t first_bit = (!A.mdirect || __ldg(A.mdirect + mdl)) ? kFirstTouch : 0u;
        Real* geo = geo_of(cur, el);
        Real* buf = buf_of(cur, el);
        uint32_t gword = 0;
        Real dd[9], lam = Real(0), mu = Real(0);
        if (active) {
            gword = ib_of(ist, el)[p];
#pragma unroll
            for (int q = 0; q < 9; ++q) dd[q] = geo[q * NN + p];
            lam = geo[9 * NN + p];
            mu = geo[10 * NN + p];
        }
        const bool on = lam != Real(0) || mu != Real(0);  // else the point adds nothing
        if (!on) {
#pragma unroll
            for (int q = 0; q < 9; ++q) dd[q] = Real(0);
        }
        __syncthreads();  // geometry stage now takes this group's old force vectors
        if (active && !(gword & first_bit)) {
            const uint32_t g = gword & kNodeMask;
#pragma unroll
            for (int d = 0; d < NFLD; ++d)
#pragma unroll
                for (int h = 0; h < CPV; ++h)
                    cp_async16(geo + (p * NFLD + d) * 4 + h * VW, A.force + ((size_t)g * NFLD + d) * 4 + h * VW);
        }
        cp_async_commit();  // group: old force of this group
        const int nxt = grp + gridDim.x;
        if (nxt < n_groups) {
            issue_gather(nxt, (it + 1) % 3, cur ^ 1);
            issue_geo(nxt, cur ^ 1);
        }
        if (nxt + (int)gridDim.x < n_groups) issue_ib(nxt + gridDim.x, (it + 2) % 3);
        cp_async_commit();  // group: next group's vectors and geometry, node table after that

        Real st[NFLD][6];
#pragma unroll
        for (int d = 0; d < NFLD; ++d)
#pragma unroll
            for (int q = 0; q < 6; ++q) st[d][q] = Real(0);
        if (active && on) {
#pragma unroll
            for (int d = 0; d < NFLD; ++d) {
                Real gx[3] = {0, 0, 0}, gy[3] = {0, 0, 0}, gz[3] = {0, 0, 0};
#pragma unroll
                for (int s = 0; s < NG; ++s) {
                    Real va[4], vb[4], vc[4];
                    load4(buf + ((((s * NG + j) * NG + k) * NFLD) + d) * 4, va);
                    load4(buf + ((((i * NG + s) * NG + k) * NFLD) + d) * 4, vb);
                    load4(buf + ((((i * NG + j) * NG + s) * NFLD) + d) * 4, vc);
                    const Real Di = sD[i * NG + s], Dj = sD[j * NG + s], Dk = sD[k * NG + s];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        gx[c] += Di * va[c];
                        gy[c] += Dj * vb[c];
                        gz[c] += Dk * vc[c];
                    }
                }
                Real gr[3][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    gr[c][0] = gx[c] * dd[0] + gy[c] * dd[1] + gz[c] * dd[2];
                    gr[c][1] = gx[c] * dd[3] + gy[c] * dd[4] + gz[c] * dd[5];
                    gr[c][2] = gx[c] * dd[6] + gy[c] * dd[7] + gz[c] * dd[8];
                }
                const Real tr = gr[0][0] + gr[1][1] + gr[2][2];
                const Real m2 = Real(2) * mu;
                st[d][0] = m2 * gr[0][0] + lam * tr;
                st[d][1] = m2 * gr[1][1] + lam * tr;
                st[d][2] = m2 * gr[2][2] + lam * tr;
                st[d][3] = m2 * (Real(0.5) * (gr[0][1] + gr[1][0]));
                st[d][4] = m2 * (Real(0.5) * (gr[0][2] + gr[2][0]));
                st[d][5] = m2 * (Real(0.5) * (gr[1][2] + gr[2][1]));
            }
        }
        __syncthreads();  // the vector buffer is reused for the fluxes
        Real r[NFLD][3];
#pragma unroll
        for (int d = 0; d < NFLD; ++d) r[d][0] = r[d][1] = r[d][2] = Real(0);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (active) {
                const Real ea = dd[a], eb = dd[3 + a], ec = dd[6 + a];
#pragma unroll
                for (int d = 0; d < NFLD; ++d)
                    store4(buf + (p * NFLD + d) * 4, st[d][0] * ea + st[d][3] * eb + st[d][4] * ec,
                           st[d][3] * ea + st[d][1] * eb + st[d][5] * ec,
                           st[d][4] * ea + st[d][5] * eb + st[d][2] * ec, Real(0));
            }
            __syncthreads();
            if (active) {
                const int ia = (a == 0) ? i : ((a == 1) ? j : k);
#pragma unroll
                for (int s = 0; s < NG; ++s) {
                    const int q = (a == 0) ? ((s * NG + j) * NG + k)
                                           : ((a == 1) ? ((i * NG + s) * NG + k) : ((i * NG + j) * NG + s));
                    const Real w = sD[s * NG + ia];
#pragma unroll
                    for (int d = 0; d < NFLD; ++d) {
                        Real v[4];
                        load4(buf + (q * NFLD + d) * 4, v);
                        r[d][0] -= w * v[0];
                        r[d][1] -= w * v[1];
                        r[d][2] -= w * v[2];
                    }
                }
            }
            if (a < 2) __syncthreads();
        }
        if (active) {
            const uint32_t g = gword & kNodeMask;
            // C-PML per cell (pml.cpp:55-216)
            const int slot = A.pml_slot ? __ldg(A.pml_slot + e) : -1;
            if (slot >= 0) {
                const double c1 = A.mc ? A.mc[mdl].c1 : A.c1, c2 = A.mc ? A.mc[mdl].c2 : A.c2;
                const Real* cf = A.pml_coef + (size_t)slot * 15 * NN + p;
                Real al[9], ab[5];
#pragma unroll
                for (int q = 0; q < 9; ++q) al[q] = __ldg(cf + q * NN);
#pragma unroll
                for (int q = 0; q < 5; ++q) ab[q] = __ldg(cf + (9 + q) * NN);
                const Real scale = __ldg(cf + 14 * NN);
                Real* mem = A.pml_mem + (size_t)slot * (3 * NFLD * 3) * NN + p;
                Real* prev = A.pml_prev + (size_t)slot * (3 * NFLD) * NN + p;
#pragma unroll
                for (int d = 0; d < NFLD; ++d) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const int f = d * 3 + c;
                        const double un = A.u[(size_t)g * 3 * NFLD + f];
                        const double vn = A.v[(size_t)g * 3 * NFLD + f];
                        const Real an = A.a[(size_t)g * 3 * NFLD + f];
                        const Real nv = Real(un + c1 * vn);
                        const Real ov = prev[f * NN] + Real(c2) * an;
                        Real m0 = mem[(f * 3 + 0) * NN], m1 = mem[(f * 3 + 1) * NN], m2 = mem[(f * 3 + 2) * NN];
                        r[d][c] += scale * (ab[0] * Real(vn) + ab[1] * Real(un) + ab[2] * m0 + ab[3] * m1 + ab[4] * m2);
                        mem[(f * 3 + 0) * NN] = al[0] * m0 + al[1] * nv + al[2] * ov;
                        mem[(f * 3 + 1) * NN] = al[3] * m1 + al[4] * nv + al[5] * ov;
                        mem[(f * 3 + 2) * NN] = al[6] * m2 + al[7] * nv + al[8] * ov;
                        prev[f * NN] = nv;
                    }
                }
            }
            // point force (solver.cpp:577-605): wavefield d takes the slots
            // of its source set, scaled by that set's source time function
            if (A.mstf) {
                int s = A.src_head ? __ldg(A.src_head + e) : -1;
                while (s >= 0) {
                    const Real w = __ldg(A.src_w + (size_t)s * NN + p);
                    const int ks = A.src_set ? __ldg(A.src_set + s) : 0;
                    if (w != Real(0)) {
#pragma unroll
                        for (int d = 0; d < NFLD; ++d) {
                            const Real stf = __ldg(A.mstf + mdl * A.n_set + A.fset[d]);
                            if (stf == Real(0) || A.fset[d] != ks) continue;
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                if (c == A.dir[d]) r[d][c] += stf * w;
                        }
                    }
                    s = __ldg(A.src_next + s);
                }
            }
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this group's old force
        __syncthreads();
        if (active) {
            const uint32_t g = gword & kNodeMask;
            const bool first = gword & first_bit;
            // the highest colour touching a node completes its force here and
            // finalises it: no cell reads the node later in this step
            const bool fin = A.fuse && (gword & kLastTouch);
#pragma unroll
            for (int d = 0; d < NFLD; ++d) {
                Real fo[4] = {Real(0), Real(0), Real(0), Real(0)};
                if (!first) load4(geo + (p * NFLD + d) * 4, fo);
                if (fin) {
                    const Real fv[3] = {fo[0] + r[d][0], fo[1] + r[d][1], fo[2] + r[d][2]};
                    const ModelConst K = A.mc ? A.mc[mdl] : ModelConst{A.nu.dt, A.nu.half_dt2, A.np.c1, A.np.c2};
                    if (A.np.coef)
                        update_node_field<Real, NFLD, true>(A.nu, A.np, g, d, fv, g < A.np.n_slot ? (int)g : -1, K);
                    else
                        update_node_field<Real, NFLD, false>(A.nu, A.np, g, d, fv, -1, K);
                } else {
                    store4(A.force + ((size_t)g * NFLD + d) * 4, fo[0] + r[d][0], fo[1] + r[d][1], fo[2] + r[d][2],
                           Real(0));
                }
            }
        }
    }
    cp_async_wait_all();
}

// ---------------------------------------------------------------------------
// elem_col_kernel: element/assembly kernel with one thread per
// (cell, wavefield, xi-line).
//
// The thread-per-point kernel above reads 15 neighbour vectors per point for
// the gradient and 15 flux vectors for the divergence, all from shared
// memory, and shared-memory bandwidth is what bounds it.  Here a thread owns
// the NG points (i = 0..NG-1, j, k) of one xi-line of one wavefield: the xi
// contractions of the gradient and of the divergence run on values held in
// registers, and only the eta and zeta neighbours go through shared memory,
// as one float per component (structure-of-arrays, no padding lane).  The
// per-(cell, wavefield) arrays are SP floats apart with SP = NG*NG (mod 32),
// so that the eta/zeta reads of a warp that spans two or three of them fall
// in distinct banks.  The D entries indexed by the loop counter come from
// the kernel parameters (constant bank); those indexed by the thread's own j
// and k are kept in registers.
//
// Pipelining: the geometry of the next group and the node table of the one
// after are bulk copies (TMA engine, one per cell, issued by one thread and
// completing on a per-stage mbarrier) into rotating shared stages; the
// writes bypass the LSU pipe that the shared-memory exchange keeps busy,
// which 16-byte cp.async by every thread did not; the next group's
// predicted-displacement vectors are register loads issued one group ahead,
// this group's old force vectors are prefetched into L2 at the start of the
// group and loaded into registers once its gradient phase is done.
// ---------------------------------------------------------------------------

// Cells per group of the line kernel: about 150 threads by default; the
// autotuner also tries the neighbouring counts at ngll 5.
__host__ __device__ constexpr int col_default_epb(int ng, int nfld) {
    return (150 / (nfld * ng * ng)) > 0 ? 150 / (nfld * ng * ng) : 1;
}

template <int NG, int NFLD, int EPB_ = col_default_epb(NG, NFLD)>
struct ColShape {
    static constexpr int NN = NG * NG * NG;
    static constexpr int NG2 = NG * NG;
    static constexpr int EPB = EPB_;                      // cells per group
    static constexpr int GR = EPB * NFLD;                 // (cell, wavefield) lines per group
    static constexpr int ACTIVE = GR * NG2;               // threads with work
    static constexpr int THREADS = (ACTIVE + 31) / 32 * 32;
    static constexpr int SP = NN + ((NG2 - NN) % 32 + 32) % 32;  // >= NN, == NG2 (mod 32)
    static constexpr int GEO_B = geo_row<float>(NN) * 4;
    static constexpr int GEO_W = GEO_B / 4;
    static constexpr int GEO_SLOT = GEO_B + 4 * (((24 - GEO_W) % 32 + 32) % 32 / 4 * 4);
    static constexpr int IB_B = ib_row_words(NN) * 4;
    static constexpr int ARR = 3 * GR * SP;               // floats of one [3][GR][SP] array
    static constexpr int N_ARR = 3;
    // dynamic shared memory without the per-model values (col_model_smem)
    static constexpr int SMEM = 2 * EPB * GEO_SLOT + 3 * EPB * IB_B + (N_ARR * ARR + 64) * 4;
    static constexpr int MIN_BLOCKS = THREADS <= 160 ? 3 : 2;
    static_assert(GEO_B % 16 == 0 && GEO_SLOT % 16 == 0 && IB_B % 16 == 0, "16-byte copies");
};

struct ColArgs {
    int e_begin, e_end, n_groups;  // range of `cells`
    const int* cells;              // the cells colour after colour
    const int* live_end;           // [colour] end of the stepping cells (several models), or null
    int colour;
    const uint32_t* ibool_padded;  // [cell][ib_row_words(NN)]: node words, model index
    const float* geom;             // [cell][geo_row]
    const float* ut;               // [node][NFLD][4]
    float* force;                  // [node][NFLD][4]
    const float* dmat;             // [NG*NG]
    const int* src_head;
    const int* src_next;
    const float* src_w;
    const float* mstf;             // [model][set] source time function value of this step
    const int* src_set;            // [slot] source set (nullptr: all set 0)
    int n_set;                     // n_model * n_set <= kMaxModels
    const int* mlive;              // [model] 1 while the model still steps
    const int* mdirect;            // [model] 1: force in full this step, 0: by increment (nullptr: in full)
    int n_model;                   // <= kMaxModels
    int dir[kMaxFields];
    int fset[kMaxFields];
    unsigned* err;                 // set to 1 when a bulk copy's wait gave up (the launch did not finish)
    float D[36];                   // D[i*NG+s], read with compile-time indices only
};

// Shared bytes of the per-model values of elem_col_kernel: source time
// function values [n_model][n_set], live and full-force flags [n_model].
__host__ __device__ constexpr int col_model_smem(int n_model, int n_set) { return (n_model * n_set + 2 * n_model) * 4; }

template <int NG, int NFLD, int EPB_>
__global__ void __launch_bounds__(ColShape<NG, NFLD, EPB_>::THREADS, ColShape<NG, NFLD, EPB_>::MIN_BLOCKS)
    elem_col_kernel(ColArgs A) {
    using S = ColShape<NG, NFLD, EPB_>;
    constexpr int NN = S::NN, NG2 = S::NG2, EPB = S::EPB, GR = S::GR, SP = S::SP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* gbase = smem_raw;
    unsigned char* ibase = gbase + 2 * EPB * S::GEO_SLOT;
    float* us = reinterpret_cast<float*>(ibase + 3 * EPB * S::IB_B);  // [3][GR][SP] displacement
    float* fe = us + S::ARR;                                          // [3][GR][SP] eta flux
    float* fz = fe + S::ARR;                                          // [3][GR][SP] zeta flux
    float* sD = us + S::N_ARR * S::ARR;

    // cells of this colour that still step (several models: the cells past
    // the last one of a live model belong to finished models)
    const int e_end = A.live_end ? min(A.e_end, A.live_end[A.colour]) : A.e_end;
    const int n_groups = e_end > A.e_begin ? (e_end - A.e_begin + EPB - 1) / EPB : 0;
    const int tid = threadIdx.x;
    const bool lane_ok = tid < S::ACTIVE;
    const int line = lane_ok ? tid / NG2 : 0;  // (cell, wavefield) line of this thread
    const int col = lane_ok ? tid - line * NG2 : 0;
    const int cl = line / NFLD, fld = line - cl * NFLD;
    const int j = col / NG, k = col - j * NG;
    int dir, fs;
    field_source<NFLD>(A.dir, A.fset, fld, dir, fs);
    // per-model step flags and source values of this step, read once per block
    // (in the dynamic shared memory after sD: col_model_smem bytes)
    float* s_stf = sD + 64;
    int* s_live = reinterpret_cast<int*>(s_stf + A.n_model * A.n_set);
    int* s_direct = s_live + A.n_model;
    for (int m = tid; m < A.n_model * A.n_set; m += S::THREADS) s_stf[m] = A.mstf[m];
    for (int m = tid; m < A.n_model; m += S::THREADS) {
        s_live[m] = A.mlive[m];
        s_direct[m] = A.mdirect ? A.mdirect[m] : 1;
    }
    if (tid < NG2) sD[tid] = A.dmat[tid];
    __syncthreads();
    float Dj[NG], Dk[NG], Tj[NG], Tk[NG];
#pragma unroll
    for (int s = 0; s < NG; ++s) {
        Dj[s] = sD[j * NG + s];
        Dk[s] = sD[k * NG + s];
        Tj[s] = sD[s * NG + j];
        Tk[s] = sD[s * NG + k];
    }

    auto geo_of = [&](int st, int c) -> const float* {
        return reinterpret_cast<const float*>(gbase + (st * EPB + c) * S::GEO_SLOT);
    };
    auto ib_of = [&](int st, int c) -> const uint32_t* {
        return reinterpret_cast<const uint32_t*>(ibase + (st * EPB + c) * S::IB_B);
    };
    // node words of this thread's line of group grp (node table in stage st)
    auto line_nodes = [&](int grp, int st, uint32_t (&w)[NG]) -> bool {
        const bool ok = lane_ok && grp < n_groups && A.e_begin + grp * EPB + cl < e_end;
#pragma unroll
        for (int i = 0; i < NG; ++i) w[i] = ok ? ib_of(st, cl)[i * NG2 + col] : 0u;
        return ok;
    };
    auto load_vectors = [&](const uint32_t (&w)[NG], bool ok, float4 (&v)[NG]) {
#pragma unroll
        for (int i = 0; i < NG; ++i)
            v[i] = ok ? __ldg(reinterpret_cast<const float4*>(A.ut) + (size_t)(w[i] & kNodeMask) * NFLD + fld)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    };

    // bulk-copy stages: barriers 0, 1 for the geometry, 2..4 for the node table
    __shared__ __align__(8) uint64_t s_bar[5];
    auto tma_geo = [&](int grp, int st) {
        if (tid != 0) return;
        const int e0 = A.e_begin + grp * EPB, nc = min(EPB, e_end - e0);
        fence_proxy_async_smem();
        mbar_expect_tx(&s_bar[st], (unsigned)(nc * S::GEO_B));
        int cell[EPB];  // looked up together
#pragma unroll
        for (int c = 0; c < EPB; ++c) cell[c] = c < nc ? __ldg(A.cells + e0 + c) : 0;
#pragma unroll
        for (int c = 0; c < EPB; ++c)
            if (c < nc)
                bulk_copy_g2s(gbase + (st * EPB + c) * S::GEO_SLOT,
                              reinterpret_cast<const unsigned char*>(A.geom) + (size_t)cell[c] * S::GEO_B, S::GEO_B, &s_bar[st]);
    };
    auto tma_ib = [&](int grp, int st) {
        if (tid != 0) return;
        const int e0 = A.e_begin + grp * EPB, nc = min(EPB, e_end - e0);
        fence_proxy_async_smem();
        mbar_expect_tx(&s_bar[2 + st], (unsigned)(nc * S::IB_B));
        int cell[EPB];
#pragma unroll
        for (int c = 0; c < EPB; ++c) cell[c] = c < nc ? __ldg(A.cells + e0 + c) : 0;
#pragma unroll
        for (int c = 0; c < EPB; ++c)
            if (c < nc)
                bulk_copy_g2s(ibase + (st * EPB + c) * S::IB_B,
                              reinterpret_cast<const unsigned char*>(A.ibool_padded) + (size_t)cell[c] * S::IB_B, S::IB_B,
                              &s_bar[2 + st]);
    };
    // a wait that gave up: flag it, give the copies in flight a second
    // bounded wait, and leave (every thread together)
    auto give_up = [&](int b0, unsigned p0, int b1, unsigned p1) {
        if (tid == 0) {
            atomicOr(A.err, 1u);
            if (b0 >= 0) mbar_wait(&s_bar[b0], p0);
            if (b1 >= 0) mbar_wait(&s_bar[b1], p1);
        }
    };

    const int G = gridDim.x;
    const int grp0 = blockIdx.x;
    if (tid == 0) {
        for (int b = 0; b < 5; ++b) mbar_init(&s_bar[b], 1);
        mbar_init_fence();
    }
    __syncthreads();
    if (grp0 < n_groups) tma_ib(grp0, 0);
    if (__syncthreads_or(grp0 < n_groups && !mbar_wait(&s_bar[2], 0))) {
        give_up(2, 0, -1, 0);
        return;
    }
    uint32_t nw[NG];
    float4 pre[NG];
    bool pre_ok = line_nodes(grp0, 0, nw);
    load_vectors(nw, pre_ok, pre);
    if (grp0 < n_groups) tma_geo(grp0, 0);
    if (grp0 + G < n_groups) tma_ib(grp0 + G, 1);

    const int ubase = line * SP + col;        // + c*GR*SP + i*NG2
    const int ebase = line * SP + col - j * NG;  // + s*NG  (eta line: i*NG2 + s*NG + k)
    const int zbase = line * SP + j * NG;        // + s     (zeta line: i*NG2 + j*NG + s)
    int it = 0;
    for (int grp = grp0; grp < n_groups; grp += G, ++it) {
        const int x = A.e_begin + grp * EPB + cl;  // of A.cells
        const int mdl = pre_ok ? (int)ib_of(it % 3, cl)[NN] : 0;
        const bool act = pre_ok && s_live[mdl];
        // first touch stores only on a full-force step; by increments
        // every touch adds to the stored force
        const uint32_t first_bit = s_direct[mdl] ? kFirstTouch : 0u;
        uint32_t cw[NG];
        float u0[NG], u1[NG], u2[NG];
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            cw[i] = nw[i];
            u0[i] = pre[i].x;
            u1[i] = pre[i].y;
            u2[i] = pre[i].z;
            if (act) {
                us[0 * GR * SP + ubase + i * NG2] = u0[i];
                us[1 * GR * SP + ubase + i * NG2] = u1[i];
                us[2 * GR * SP + ubase + i * NG2] = u2[i];
            }
        }
        const int nx = grp + G;
        {
            // stage it&1 holds this group's geometry (use it/2 of that stage),
            // stage (it+1)%3 the next group's node table (use (it+1)/3)
            const unsigned pg = (unsigned)(it >> 1) & 1u, pi = (unsigned)((it + 1) / 3) & 1u;
            const int bi = nx < n_groups ? 2 + (it + 1) % 3 : -1;
            bool bad = !mbar_wait(&s_bar[it & 1], pg);
            if (bi >= 0) bad = !mbar_wait(&s_bar[bi], pi) || bad;
            if (__syncthreads_or(bad)) {  // displacement of this group, its geometry, the next node table
                give_up(it & 1, pg, bi, pi);
                return;
            }
        }
        if (nx < n_groups) tma_geo(nx, (it + 1) & 1);
        if (nx + G < n_groups) tma_ib(nx + G, (it + 2) % 3);
        // old force vectors of the nodes this colour does not touch first:
        // start their DRAM reads into L2 now, so the loads issued after the
        // flux phase find them there (no registers held meanwhile)
        if (act) {
#pragma unroll
            for (int i = 0; i < NG; ++i)
                if (!(cw[i] & first_bit)) {
                    const float4* pf = reinterpret_cast<const float4*>(A.force) + (size_t)(cw[i] & kNodeMask) * NFLD + fld;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(pf));
                }
        }
        const float stf = act ? s_stf[mdl * A.n_set + fs] : 0.f;
        const int src = (act && stf != 0.f && A.src_head) ? __ldg(A.src_head + __ldg(A.cells + x)) : -1;
        pre_ok = line_nodes(nx, (it + 1) % 3, nw);
        load_vectors(nw, pre_ok, pre);

        // old force of the nodes this colour does not touch first
        float4 of[NG];
        auto load_old_force = [&]() {
#pragma unroll
            for (int i = 0; i < NG; ++i)
                of[i] = (act && !(cw[i] & first_bit))
                            ? *(reinterpret_cast<const float4*>(A.force) + (size_t)(cw[i] & kNodeMask) * NFLD + fld)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        // gradient, stress and the three fluxes at each point of the line
        float fx0[NG], fx1[NG], fx2[NG];
        const float* geo = geo_of(it & 1, cl);
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            fx0[i] = fx1[i] = fx2[i] = 0.f;
            if (!act) continue;
            const int p = i * NG2 + col;
            float dd[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) dd[q] = geo[q * NN + p];
            const float lam = geo[9 * NN + p], mu = geo[10 * NN + p];
            float gx[3] = {0.f, 0.f, 0.f}, gy[3] = {0.f, 0.f, 0.f}, gz[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < NG; ++s) {
                const float Di = A.D[i * NG + s];
                gx[0] += Di * u0[s];
                gx[1] += Di * u1[s];
                gx[2] += Di * u2[s];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float* uc = us + c * GR * SP + i * NG2;
#pragma unroll
                for (int s = 0; s < NG; ++s) {
                    gy[c] += Dj[s] * uc[ebase + s * NG];
                    gz[c] += Dk[s] * uc[zbase + s];
                }
            }
            float gr[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gr[c][0] = gx[c] * dd[0] + gy[c] * dd[1] + gz[c] * dd[2];
                gr[c][1] = gx[c] * dd[3] + gy[c] * dd[4] + gz[c] * dd[5];
                gr[c][2] = gx[c] * dd[6] + gy[c] * dd[7] + gz[c] * dd[8];
            }
            const float tr = gr[0][0] + gr[1][1] + gr[2][2];
            const float m2 = 2.f * mu;
            const float st0 = m2 * gr[0][0] + lam * tr;
            const float st1 = m2 * gr[1][1] + lam * tr;
            const float st2 = m2 * gr[2][2] + lam * tr;
            const float st3 = mu * (gr[0][1] + gr[1][0]);
            const float st4 = mu * (gr[0][2] + gr[2][0]);
            const float st5 = mu * (gr[1][2] + gr[2][1]);
            // flux along axis a: sigma . (dd[a], dd[3+a], dd[6+a]); 0 where the
            // point adds nothing
            const bool on = lam != 0.f || mu != 0.f;
            auto flux = [&](float a, float b, float c, int x) {
                return on ? a * dd[x] + b * dd[3 + x] + c * dd[6 + x] : 0.f;
            };
            fx0[i] = flux(st0, st3, st4, 0);
            fx1[i] = flux(st3, st1, st5, 0);
            fx2[i] = flux(st4, st5, st2, 0);
            const float e0 = flux(st0, st3, st4, 1), e1 = flux(st3, st1, st5, 1), e2 = flux(st4, st5, st2, 1);
            const float z0 = flux(st0, st3, st4, 2), z1 = flux(st3, st1, st5, 2), z2 = flux(st4, st5, st2, 2);
            fe[0 * GR * SP + ubase + i * NG2] = e0;
            fe[1 * GR * SP + ubase + i * NG2] = e1;
            fe[2 * GR * SP + ubase + i * NG2] = e2;
            fz[0 * GR * SP + ubase + i * NG2] = z0;
            fz[1 * GR * SP + ubase + i * NG2] = z1;
            fz[2 * GR * SP + ubase + i * NG2] = z2;
        }
        load_old_force();
        __syncthreads();  // fluxes of the whole group
        if (act) {
#pragma unroll
            for (int i = 0; i < NG; ++i) {
                const int p = i * NG2 + col;
                float r[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int s = 0; s < NG; ++s) {
                    const float Ti = A.D[s * NG + i];
                    r[0] += Ti * fx0[s];
                    r[1] += Ti * fx1[s];
                    r[2] += Ti * fx2[s];
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float* ec = fe + c * GR * SP + i * NG2;
                    const float* zc = fz + c * GR * SP + i * NG2;
#pragma unroll
                    for (int s = 0; s < NG; ++s) {
                        r[c] += Tj[s] * ec[ebase + s * NG];
                        r[c] += Tk[s] * zc[zbase + s];
                    }
                }
                r[0] = -r[0];
                r[1] = -r[1];
                r[2] = -r[2];
                // point force (solver.cpp:577-605)
                for (int sl = src; sl >= 0; sl = __ldg(A.src_next + sl)) {
                    if (A.src_set && __ldg(A.src_set + sl) != fs) continue;
                    const float w = __ldg(A.src_w + (size_t)sl * NN + p);
                    if (w != 0.f) {
                        const float sw = stf * w;
                        if (dir == 0) r[0] += sw;
                        else if (dir == 1) r[1] += sw;
                        else r[2] += sw;
                    }
                }
                float4* dst = reinterpret_cast<float4*>(A.force) + (size_t)(cw[i] & kNodeMask) * NFLD + fld;
                *dst = make_float4(of[i].x + r[0], of[i].y + r[1], of[i].z + r[2], 0.f);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// elem_gather_kernel: the element kernel of the time loop (both precisions).
//
// A group of WARPS warps takes CELLS cells at a time and leaves their force
// contributions in contrib; the node pass adds them up (NodeGather).  Against a
// read-modify-write of the assembled force colour after colour this stores 4 (8)
// bytes per value in whole rows instead of reading and writing 16-byte vectors
// node by node, needs one launch instead of one per colour, and takes the cells
// in mesh order, so the predicted displacement of the nodes that neighbours
// share comes from L2.
//
// One thread per xi-line: the NG points (i = 0..NG-1, j, k) of a cell, for one
// wavefield after the other, so the geometry is fetched once for all of them
// and the wavefield count is a run-time value.  The xi contractions run on
// registers.  For the eta and zeta contractions the thread with column (j, k)
// also owns the eta line (i = j, k) and the zeta line (i = k, j): it reads the
// line from shared memory, contracts it with D (constant bank) and writes the
// result back in place.  Phases per wavefield: own displacements into both
// arrays | line contractions | gradient, stress, fluxes in place | line
// contractions | divergence and store.  With one warp per group (NG <= 5; 25
// of 32 lanes at NG = 5) the phases are separated by warp-level barriers only
// and the warps of a block run independently, which hides the exchange's
// latency better than full lanes behind block barriers.
//
// A group's geometry is a bulk copy (TMA engine) on an mbarrier, issued as
// soon as the last wavefield of the previous group has read the stage; the
// node words two groups and the displacement vectors one wavefield ahead are
// register loads.  The contributions of a chunk of wavefields are collected in
// shared memory and leave as one bulk store per cell.
//
// Measured on 40 x 40 x 20 cells of ngll 5: FP32 with three wavefields 205 us
// (3,780 instructions and 1,020 shared wavefronts per cell, the L1 pipe 69 %
// busy, issue 57 %, DRAM 24 %); by colour the same took about 310 us.  FP64
// with one wavefield 136 us.
// ---------------------------------------------------------------------------

// Point (i, j, k) of an exchange array at P*i + NG*j + k, a cell's component
// S words apart (eta: PE, SE; zeta: PZ, SZ), chosen by enumeration so that a
// warp's own-point and line accesses fall in distinct banks (4-byte words) or
// nearly so (8-byte words).
template <int NG, bool WIDE>
struct GatherPad;
template <> struct GatherPad<3, false> { static constexpr int PE = 14, SE = 43, PZ = 27, SZ = 73; };
template <> struct GatherPad<3, true> { static constexpr int PE = 19, SE = 57, PZ = 17, SZ = 57; };
template <> struct GatherPad<4, false> { static constexpr int PE = 20, SE = 80, PZ = 17, SZ = 80; };
template <> struct GatherPad<4, true> { static constexpr int PE = 20, SE = 76, PZ = 17, SZ = 67; };
template <> struct GatherPad<5, false> { static constexpr int PE = 26, SE = 130, PZ = 25, SZ = 125; };
template <> struct GatherPad<5, true> { static constexpr int PE = 26, SE = 130, PZ = 26, SZ = 130; };
template <> struct GatherPad<6, false> { static constexpr int PE = 38, SE = 228, PZ = 49, SZ = 292; };
template <> struct GatherPad<6, true> { static constexpr int PE = 38, SE = 228, PZ = 41, SZ = 244; };

template <typename Real, int NG>
struct GatherShape : GatherPad<NG, sizeof(Real) == 8> {
    using Pad = GatherPad<NG, sizeof(Real) == 8>;
    static constexpr int NN = NG * NG * NG, NG2 = NG * NG;
    static constexpr int WARPS = NG2 <= 32 ? 1 : 4;        // warps of a group
    static constexpr int CELLS = WARPS * 32 / NG2;         // cells of a group
    static constexpr int GROUPS = WARPS == 1 ? 4 : 1;      // groups of a block
    static constexpr int THREADS = 32 * WARPS * GROUPS;
    static constexpr int GEO_B = geo_row<Real>(NN) * (int)sizeof(Real);
    // several cells per warp: their rows NG2 words apart modulo the banks
    static constexpr int SKEW = CELLS == 1 ? 0 : ((NG2 * (int)sizeof(Real) - GEO_B) % 128 + 128) % 128 / 16 * 16;
    static constexpr int GEO_SLOT = GEO_B + SKEW;
    static constexpr int XCH_B = (3 * CELLS * (Pad::SE + Pad::SZ) * (int)sizeof(Real) + 15) / 16 * 16;
    // contributions on their way out (FP64: in the eta array, which is free by then)
    static constexpr int CHUNK_MAX_B = gather_chunk_units<Real>(NN, 3) * 3 * (int)sizeof(Real);
    static constexpr bool OUT_IN_XCH = sizeof(Real) == 8;
    static_assert(!OUT_IN_XCH || CHUNK_MAX_B <= 3 * Pad::SE * (int)sizeof(Real), "a chunk fits in the eta array");
    static constexpr int GROUP_B = CELLS * GEO_SLOT + XCH_B + (OUT_IN_XCH ? 0 : CELLS * CHUNK_MAX_B);
    static constexpr int SMEM = GROUPS * GROUP_B;
    // at most 128 registers a thread in FP32, 168 in FP64
    static constexpr int MIN_BLOCKS = (sizeof(Real) == 4 ? 608 : 384) / THREADS;
};

template <typename Real>
struct GatherArgs {
    int n_cell;
    const int* live_end;           // [1] end of the stepping cells (several models), or null
    const uint32_t* ibool_padded;  // [cell][ib_row_words(NN)]: node words, model index
    const Real* geom;              // [cell][geo_row]
    const Real* ut;                // [node][nfld][4]
    Real* contrib;                 // [cell][chunk][NN][chunk's fields][3]
    int nfld;                      // wavefields
    int nfld_item;                 // wavefields of one work item: nfld, or 1 where the cells alone are too few
    const int* mlive;              // [model]
    bool multi;                    // several models
    // source
    const int* src_head;
    const int* src_next;
    const Real* src_w;
    const Real* mstf;              // [model][set] source time function value of this step
    const int* src_set;
    int n_set;
    int dir[kMaxFields];
    int fset[kMaxFields];
    unsigned* err;                 // set to 1 when a bulk copy's wait gave up (the launch did not finish)
    Real D[36];                    // D[i*NG+s], read with compile-time indices only
    float2 D2[36];                 // the same twice, for packed operations (FP32)
};

// C-PML per cell (pml.cpp:55-216), after the element kernel: the term with
// last step's memory is added to the cells' contributions, and the memory
// moves on, which only uses values fixed at the start of the step.  A block
// takes a C-PML cell at a time, one thread per (component, point); the arrays
// are streams of whole rows.  An axis that is live nowhere in a cell (its A_k
// are 0 there) has a memory nothing reads: it is neither loaded nor updated,
// which is more than half of the traffic in the one-axis cells that most C-PML
// cells are.  Inside the element
// kernel, with 12 warps per SM and every axis, the same work took 220 us on
// 40 x 40 x 20 cells (15,600 of them C-PML, FP64, one wavefield).
template <typename Real>
struct CellPmlArgs {
    int n_slot;
    const int2* cell;              // [slot] cell, live axes (bits 0..2)
    const uint32_t* ibool_padded;
    Real* contrib;
    int nfld;
    const int* mlive;
    bool multi;                    // several models
    const Real* coef;              // [slot][15][NN]
    Real* mem;                     // [slot][9*nfld][NN]
    Real* prev;                    // [slot][3*nfld][NN]
    const double* u;               // [node][3*nfld]
    const double* v;
    const Real* a;
    const ModelConst* mc;          // [model]
};

constexpr int cell_pml_threads(int nn) { return (3 * nn + 31) / 32 * 32; }
// Threads per SM, for 80 registers: with 1280 (56 registers, spills) the pass
// takes 164 us on the mesh above, with 768 about 139 (575 MB of DRAM traffic).
constexpr int kCellPmlThreads = 768;

// EARLY: launched before the element kernel has completed; the first cell's
// coefficients are on their way while that ends.
template <typename Real, int NG, bool EARLY>
__global__ void __launch_bounds__(cell_pml_threads(NG * NG * NG), kCellPmlThreads / cell_pml_threads(NG * NG * NG))
    cell_pml_kernel(const __grid_constant__ CellPmlArgs<Real> A) {
    constexpr int NN = NG * NG * NG;
    const int F = 3 * A.nfld, fc = gather_chunk_fields<Real>(A.nfld);
    const int chunk_u = gather_chunk_units<Real>(NN, A.nfld);
    const int c = threadIdx.x / NN, p = threadIdx.x - c * NN;
    const int step = gridDim.x;
    auto cell_at = [&](int slot) { return slot < A.n_slot ? __ldg(A.cell + slot) : make_int2(0, 0); };
    auto node_at = [&](int cell) { return c < 3 ? __ldg(A.ibool_padded + (size_t)cell * ib_row_words(NN) + p) & kNodeMask : 0u; };
    int2 ce = cell_at(blockIdx.x);
    uint32_t g = node_at(ce.x);
    bool first = EARLY;  // the grid leaves no block without a slot
    if (!EARLY) {
        pdl_wait();
        pdl_launch();
    }
    for (int slot = blockIdx.x; slot < A.n_slot; slot += step) {
        // the next cell's index and nodes are on their way during this one
        const int2 ce1 = cell_at(slot + step);
        const int mdl = A.multi ? (int)__ldg(A.ibool_padded + (size_t)ce.x * ib_row_words(NN) + NN) : 0;
        bool on = c < 3 && ((EARLY && first) || __ldcg(A.mlive + mdl));
        Real scale = Real(0), b0 = Real(0), b1 = Real(0), bq[3], al[3][3];
        auto load_coef = [&]() {
            const Real* cf = A.coef + (size_t)slot * 15 * NN + p;
            scale = __ldg(cf + 14 * NN), b0 = __ldg(cf + 9 * NN), b1 = __ldg(cf + 10 * NN);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const bool live = ce.y >> q & 1;
                bq[q] = live ? __ldg(cf + (11 + q) * NN) : Real(0);
#pragma unroll
                for (int x = 0; x < 3; ++x) al[q][x] = live ? __ldg(cf + (3 * q + x) * NN) : Real(0);
            }
        };
        if (EARLY && on) load_coef();
        if (EARLY && first) {
            pdl_wait();
            pdl_launch();
            on = on && __ldcg(A.mlive + mdl);
        }
        if (on) {
            if (!EARLY) load_coef();
            const size_t at = (size_t)g * F + c;
            const double k1 = A.mc[mdl].c1;
            const Real k2 = (Real)A.mc[mdl].c2;
            for (int d = 0; d < A.nfld; ++d) {
                Real* mem = A.mem + ((size_t)slot * 3 * F + 9 * d + 3 * c) * NN + p;
                Real* prev = A.prev + ((size_t)slot * F + 3 * d + c) * NN + p;
                Real* out = A.contrib + ((size_t)ce.x * (A.nfld / fc) * chunk_u + (size_t)(d / fc) * chunk_u + p * fc + d % fc) * 3 + c;
                // the rows that come from DRAM first: 374 us per step against 379
                // with the state's loads first (40 x 40 x 20 cells, FP64)
                Real m[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) m[q] = ce.y >> q & 1 ? mem[q * NN] : Real(0);
                const Real old = *out;
                const Real pr = *prev, an = A.a[at + 3 * d];
                const double un = A.u[at + 3 * d], vn = A.v[at + 3 * d];
                const Real nv = Real(un + k1 * vn), ov = pr + k2 * an;
                Real r = b0 * Real(vn) + b1 * Real(un);
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (ce.y >> q & 1) {
                        r += bq[q] * m[q];
                        mem[q * NN] = al[q][0] * m[q] + al[q][1] * nv + al[q][2] * ov;
                    }
                *prev = nv;
                *out = old + scale * r;
            }
        }
        first = false;
        ce = ce1;
        g = node_at(ce.x);
    }
}

// Packed pairs of FP32 operations (one instruction for two, sm_100) beside the
// plain ones, so that one expression serves two points or one.
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double vmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
// One value, or two that lie `step` apart.
template <typename Real>
__device__ __forceinline__ void vload(const Real* p, int, Real& x) { x = p[0]; }
__device__ __forceinline__ void vload(const float* p, int step, float2& x) { x = make_float2(p[0], p[step]); }
template <typename Real>
__device__ __forceinline__ void vstore(Real* p, int, Real x) { p[0] = x; }
__device__ __forceinline__ void vstore(float* p, int step, float2 x) { p[0] = x.x, p[step] = x.y; }
__device__ __forceinline__ float2 vpair(float a, float b) { return make_float2(a, b); }
// x where a or b is not 0, else 0 (also if x is not a number)
template <typename Real>
__device__ __forceinline__ Real vwhere(Real a, Real b, Real x) { return a != Real(0) || b != Real(0) ? x : Real(0); }
__device__ __forceinline__ float2 vwhere(float2 a, float2 b, float2 x) {
    return make_float2(vwhere(a.x, b.x, x.x), vwhere(a.y, b.y, x.y));
}

// Gradient to fluxes at one point (V = Real) or, in FP32, two (float2) whose
// geometry lies `step` apart: g[c][b] the derivatives of component c along
// reference axis b; fl[b][c] the flux along axis b.  OFF: 0 at the points that add
// nothing (lambda and mu stored as 0), where a collapsed cell's infinite dxi_dx
// would otherwise make 0 * inf of it.
template <bool OFF, typename Real, typename V>
__device__ __forceinline__ void point_fluxes(const Real* geo, int nn, int step, const V (&g)[3][3], V (&fl)[3][3]) {
    V dd[9], lam, mu, gr[3][3];
#pragma unroll
    for (int x = 0; x < 9; ++x) vload(geo + x * nn, step, dd[x]);
    vload(geo + 9 * nn, step, lam);
    vload(geo + 10 * nn, step, mu);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a)
            gr[c][a] = vfma(g[c][2], dd[3 * a + 2], vfma(g[c][1], dd[3 * a + 1], vmul(g[c][0], dd[3 * a])));
    const V tr = vmul(lam, vadd(vadd(gr[0][0], gr[1][1]), gr[2][2]));
    const V m2 = vadd(mu, mu);
    V st[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) st[c][c] = vfma(m2, gr[c][c], tr);
    st[0][1] = st[1][0] = vmul(mu, vadd(gr[0][1], gr[1][0]));
    st[0][2] = st[2][0] = vmul(mu, vadd(gr[0][2], gr[2][0]));
    st[1][2] = st[2][1] = vmul(mu, vadd(gr[1][2], gr[2][1]));
    // flux along axis b: sigma . (dd[b], dd[3+b], dd[6+b])
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            fl[b][c] = vfma(st[c][2], dd[6 + b], vfma(st[c][1], dd[3 + b], vmul(st[c][0], dd[b])));
            if (OFF) fl[b][c] = vwhere(lam, mu, fl[b][c]);
        }
}

template <typename Real, int NG>
__global__ void __launch_bounds__(GatherShape<Real, NG>::THREADS, GatherShape<Real, NG>::MIN_BLOCKS)
    elem_gather_kernel(const __grid_constant__ GatherArgs<Real> A) {
    using S = GatherShape<Real, NG>;
    constexpr int NN = S::NN, NG2 = S::NG2, CELLS = S::CELLS, PE = S::PE, SE = S::SE, PZ = S::PZ, SZ = S::SZ;
    constexpr int IB_W = ib_row_words(NN);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_bar[S::GROUPS];
    const int gid = threadIdx.x / (32 * S::WARPS), gt = threadIdx.x - gid * 32 * S::WARPS;
    unsigned char* geo_b = smem_raw + gid * S::GROUP_B;
    Real* xe = reinterpret_cast<Real*>(geo_b + CELLS * S::GEO_SLOT);  // [3][CELLS][SE]
    Real* xz = xe + 3 * CELLS * SE;                                   // [3][CELLS][SZ]
    Real* stage = S::OUT_IN_XCH ? xe : reinterpret_cast<Real*>(geo_b + CELLS * S::GEO_SLOT + S::XCH_B);
    uint64_t* bar = s_bar + gid;
    auto sync = [&]() {
        if constexpr (S::WARPS == 1) __syncwarp();
        else __syncthreads();
    };
    auto any = [&](bool x) -> bool {
        if constexpr (S::WARPS == 1) return __any_sync(0xffffffffu, x);
        else return __syncthreads_or(x);
    };
    if (gt == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    __syncthreads();

    const bool lane_ok = gt < CELLS * NG2;
    const int cl = lane_ok ? gt / NG2 : 0;
    const int col = lane_ok ? gt - cl * NG2 : 0;
    const int j = col / NG, k = col - j * NG;
    if (A.live_end) pdl_wait();
    const int n_cell = A.live_end ? min(A.n_cell, __ldcg(A.live_end)) : A.n_cell;
    const int split = A.nfld / A.nfld_item;
    const int fc = gather_chunk_fields<Real>(A.nfld), chunk_u = gather_chunk_units<Real>(NN, A.nfld);
    const bool staged = A.nfld_item % fc == 0;  // an item fills whole chunks
    const size_t row_u = (size_t)(A.nfld / fc) * chunk_u;
    const int n_item = (n_cell + CELLS - 1) / CELLS * split;
    const int step = gridDim.x * S::GROUPS;
    const int first = blockIdx.x * S::GROUPS + gid;
    const Real* geo = reinterpret_cast<const Real*>(geo_b + cl * S::GEO_SLOT);
    const int own_e = cl * SE + col, own_z = cl * SZ + col;            // + i*PE, i*PZ
    const int line_e = cl * SE + j * PE + k, line_z = cl * SZ + k * PZ + j * NG;  // + s*NG, + s

    auto copy_geo = [&](int item) {
        if (gt != 0) return;
        const int e0 = item / split * CELLS, nc = min(CELLS, n_cell - e0);
        fence_proxy_async_smem();
        mbar_expect_tx(bar, (unsigned)(nc * S::GEO_B));
        for (int c = 0; c < nc; ++c)
            bulk_copy_g2s(geo_b + c * S::GEO_SLOT, A.geom + (size_t)(e0 + c) * geo_row<Real>(NN), S::GEO_B, bar);
    };
    auto cell_of = [&](int item) -> int {  // this thread's cell, -1 without one
        const int e = item / split * CELLS + cl;
        return lane_ok && item < n_item && e < n_cell ? e : -1;
    };
    auto load_words = [&](int item, uint32_t (&w)[NG]) {
        const int e = cell_of(item);
#pragma unroll
        for (int i = 0; i < NG; ++i) w[i] = e >= 0 ? __ldg(A.ibool_padded + (size_t)e * IB_W + i * NG2 + col) : 0u;
    };
    auto load_vectors = [&](const uint32_t (&w)[NG], bool ok, int d, Real (&x)[3][NG]) {
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const Real* src = A.ut + ((size_t)(w[i] & kNodeMask) * A.nfld + d) * 4;
            if constexpr (sizeof(Real) == 4) {
                const float4 t = ok ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[0][i] = t.x, x[1][i] = t.y, x[2][i] = t.z;
            } else {
                const double2 t = ok ? *reinterpret_cast<const double2*>(src) : make_double2(0.0, 0.0);
                x[0][i] = t.x, x[1][i] = t.y, x[2][i] = ok ? src[2] : 0.0;
            }
        }
    };

    uint32_t nw[NG], nw2[NG];  // node words: the next item's, the one's after
    Real pre[3][NG];                   // displacement of the wavefield to come
    load_words(first, nw);
    load_words(first + step, nw2);
    if (first < n_item) copy_geo(first);
    pdl_wait();
    pdl_launch();
    load_vectors(nw, cell_of(first) >= 0, first % split * A.nfld_item, pre);
    unsigned phase = 0;
    for (int item = first; item < n_item; item += step) {
        const int e = cell_of(item), next = item + step;
        const int mdl = A.multi && e >= 0 ? (int)__ldg(A.ibool_padded + (size_t)e * IB_W + NN) : 0;
        const bool act = e >= 0 && __ldcg(A.mlive + mdl) != 0;
        const int src0 = act && A.src_head ? __ldg(A.src_head + e) : -1;
#pragma unroll
        for (int i = 0; i < NG; ++i) nw[i] = nw2[i];
        load_words(next + step, nw2);
        if (any(!mbar_wait(bar, phase))) {
            // the copy never came: flag it, give it a second bounded wait, let
            // the stores on their way read their shared memory, leave
            if (gt == 0) {
                atomicOr(A.err, 1u);
                mbar_wait(bar, phase);
                bulk_wait_all();
            }
            return;
        }
        phase ^= 1u;
        const int d0 = item % split * A.nfld_item, d1 = d0 + A.nfld_item;
        for (int d = d0; d < d1; ++d) {
            Real u[3][NG];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int i = 0; i < NG; ++i) {
                    u[c][i] = pre[c][i];
                    if (lane_ok) {
                        xe[c * CELLS * SE + own_e + i * PE] = u[c][i];
                        xz[c * CELLS * SZ + own_z + i * PZ] = u[c][i];
                    }
                }
            sync();
            if (d + 1 < d1) {
                uint32_t w[NG];
                load_words(item, w);
                load_vectors(w, e >= 0, d + 1, pre);
            } else {
                load_vectors(nw, cell_of(next) >= 0, next % split * A.nfld_item, pre);
            }
            // the eta and zeta derivatives along this thread's lines, in place
            // (FP32: the two lines as one packed pair)
            auto contract = [&](auto index) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    Real* le = xe + c * CELLS * SE + line_e;
                    Real* lz = xz + c * CELLS * SZ + line_z;
                    if constexpr (sizeof(Real) == 4) {
                        float2 v[NG];
#pragma unroll
                        for (int t = 0; t < NG; ++t) v[t] = vpair(le[t * NG], lz[t]);
#pragma unroll
                        for (int s2 = 0; s2 < NG; ++s2) {
                            float2 x = vmul(A.D2[index(s2, 0)], v[0]);
#pragma unroll
                            for (int t = 1; t < NG; ++t) x = vfma(A.D2[index(s2, t)], v[t], x);
                            le[s2 * NG] = x.x;
                            lz[s2] = x.y;
                        }
                    } else {
                        Real ve[NG], vz[NG];
#pragma unroll
                        for (int t = 0; t < NG; ++t) {
                            ve[t] = le[t * NG];
                            vz[t] = lz[t];
                        }
#pragma unroll
                        for (int s2 = 0; s2 < NG; ++s2) {
                            Real de = Real(0), dz = Real(0);
#pragma unroll
                            for (int t = 0; t < NG; ++t) {
                                de += A.D[index(s2, t)] * ve[t];
                                dz += A.D[index(s2, t)] * vz[t];
                            }
                            le[s2 * NG] = de;
                            lz[s2] = dz;
                        }
                    }
                }
            };
            if (lane_ok) contract([&](int s2, int t) { return s2 * NG + t; });
            sync();
            // gradient, stress and the three fluxes at each point of the line
            Real fx[3][NG];
            if (lane_ok) {
                auto xi = [&](int c, int i) -> Real {
                    Real x = A.D[i * NG] * u[c][0];
#pragma unroll
                    for (int s = 1; s < NG; ++s) x = vfma(A.D[i * NG + s], u[c][s], x);
                    return x;
                };
                // at points i and, in pairs, i + 1 (FP32: two at a time)
                auto fluxes = [&](auto zero, int i) {
                    using V = decltype(zero);
                    V g[3][3], fl[3][3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if constexpr (sizeof(V) > sizeof(Real)) g[c][0] = vpair(xi(c, i), xi(c, i + 1));
                        else g[c][0] = xi(c, i);
                        vload(xe + c * CELLS * SE + own_e + i * PE, PE, g[c][1]);
                        vload(xz + c * CELLS * SZ + own_z + i * PZ, PZ, g[c][2]);
                    }
                    point_fluxes<true>(geo + i * NG2 + col, NN, NG2, g, fl);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if constexpr (sizeof(V) > sizeof(Real)) {
                            fx[c][i] = fl[0][c].x;
                            fx[c][i + 1] = fl[0][c].y;
                        } else {
                            fx[c][i] = fl[0][c];
                        }
                        vstore(xe + c * CELLS * SE + own_e + i * PE, PE, fl[1][c]);
                        vstore(xz + c * CELLS * SZ + own_z + i * PZ, PZ, fl[2][c]);
                    }
                };
                constexpr int PAIRS = sizeof(Real) == 4 ? NG / 2 : 0;
                if constexpr (PAIRS > 0) {
#pragma unroll
                    for (int h = 0; h < PAIRS; ++h) fluxes(float2{}, 2 * h);
                }
#pragma unroll
                for (int i = 2 * PAIRS; i < NG; ++i) fluxes(Real(0), i);
            }
            sync();  // and the geometry has been read
            if (d + 1 == d1 && next < n_item) copy_geo(next);
            if (lane_ok) contract([&](int s2, int t) { return t * NG + s2; });
            if (gt == 0) bulk_wait_read();  // the chunk before has left the stage
            sync();
            Real r[3][NG];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int i = 0; i < NG; ++i) {
                    Real x = Real(0);
#pragma unroll
                    for (int s = 0; s < NG; ++s) x += A.D[s * NG + i] * fx[c][s];
                    x += xe[c * CELLS * SE + own_e + i * PE];
                    x += xz[c * CELLS * SZ + own_z + i * PZ];
                    r[c][i] = -x;
                }
            // point force (solver.cpp:577-605)
            if (src0 >= 0 && A.mstf) {
                const int fs = A.fset[d], dir = A.dir[d];
                const Real stf = __ldcg(A.mstf + mdl * A.n_set + fs);
                for (int sl = stf != Real(0) ? src0 : -1; sl >= 0; sl = __ldg(A.src_next + sl)) {
                    if (A.src_set && __ldg(A.src_set + sl) != fs) continue;
#pragma unroll
                    for (int i = 0; i < NG; ++i) {
                        const Real sw = stf * __ldg(A.src_w + (size_t)sl * NN + i * NG2 + col);
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            if (c == dir) r[c][i] += sw;
                    }
                }
            }
            const int dc = d % fc;
            if (!staged) {
                if (act) {
                    Real* out = A.contrib + ((size_t)e * row_u + (size_t)(d / fc) * chunk_u + col * fc + dc) * 3;
#pragma unroll
                    for (int i = 0; i < NG; ++i)
#pragma unroll
                        for (int c = 0; c < 3; ++c) out[i * NG2 * fc * 3 + c] = r[c][i];
                }
                continue;
            }
            if constexpr (S::OUT_IN_XCH) sync();  // every thread has read the eta array
            if (lane_ok) {
                Real* out = stage + (cl * chunk_u + col * fc + dc) * 3;
#pragma unroll
                for (int i = 0; i < NG; ++i)
#pragma unroll
                    for (int c = 0; c < 3; ++c) out[i * NG2 * fc * 3 + c] = r[c][i];
            }
            if (dc + 1 == fc) {
                fence_proxy_async_smem();
                sync();
                if (gt == 0) {
                    const int e0 = item / split * CELLS, nc = min(CELLS, n_cell - e0);
                    for (int c = 0; c < nc; ++c)
                        bulk_copy_s2g(A.contrib + ((size_t)(e0 + c) * row_u + (size_t)(d / fc) * chunk_u) * 3,
                                      stage + c * chunk_u * 3, (unsigned)(chunk_u * 3 * sizeof(Real)));
                    bulk_commit();
                    if constexpr (S::OUT_IN_XCH) bulk_wait_read();
                }
                if constexpr (S::OUT_IN_XCH) sync();
            }
        }
    }
    if (gt == 0) bulk_wait_all();
}

// ---------------------------------------------------------------------------
// elem_plane_kernel: the gather kernel's work for wavefields in threes at
// ngll 5 in FP32, one thread per xi-plane.
//
// A warp takes two cells and three wavefields: lane (cell, wavefield, i) owns
// the 25 points (i, j, k) of one plane, with their displacement and the
// residual it accumulates in registers, so the eta and zeta contractions, of
// the gradient and of the divergence, touch no shared memory.  Only the xi
// contractions exchange: lane (., i) also owns the five xi-lines of row j = i,
// in place in one array.  Against one thread per xi-line (two directions
// exchanged, 25 of 32 lanes) that halves the shared-memory accesses and takes
// 30 of 32 lanes: 2,400 instructions and 580 shared wavefronts per cell
// against 3,780 and 1,020.  It runs 8 warps per SM (255 registers), which the
// independent work of 25 points per thread does not quite make up for (issue
// slots 43 % busy; waits for the gathers, FMA latency and instruction fetch
// on top): 32,000 cells x 3 wavefields take 173 us against 205, DRAM 25 %
// busy in both.  Pairs of points use packed FP32 operations (2,900
// instructions and 190 us without).  Point (i, j, k) of (cell, wavefield) q sits
// at 135 q + 27 i + 5 j + k: a warp's own-point and line accesses fall in
// distinct banks.  Node words come by bulk copy one item ahead, the geometry
// as soon as the last one has been read; the contributions leave as one bulk
// copy per cell, collected in the exchange array.  OFF: the mesh has points with
// mu <= 0; the selects at every point cost 1.2 % of a step (404 against 399 us,
// same cells), which the line kernel hides.
// ---------------------------------------------------------------------------
struct PlaneShape {
    static constexpr int NG = 5, NN = 125, NG2 = 25, CELLS = 2, WARPS = 4, THREADS = 32 * WARPS;
    static constexpr int PI = 27, SQ = 135, SC = 6 * SQ;  // words between planes, (cell, wavefield)s, components
    static constexpr int GEO_B = geo_row<float>(NN) * 4;
    static constexpr int GEO_SLOT = GEO_B + 48;            // 12 banks apart
    static constexpr int IB_B = ib_row_words(NN) * 4;
    static constexpr int CHUNK_W = gather_chunk_units<float>(NN, 3) * 3;
    static constexpr int XCH_B = (3 * SC * 4 + 15) / 16 * 16;
    static constexpr int WARP_B = CELLS * GEO_SLOT + 2 * CELLS * IB_B + XCH_B;
    static constexpr int SMEM = WARPS * WARP_B;
    static_assert(CELLS * CHUNK_W * 4 <= XCH_B, "the contributions fit in the exchange array");
};

template <bool OFF>
static __global__ void __launch_bounds__(PlaneShape::THREADS, 2)
    elem_plane_kernel(const __grid_constant__ GatherArgs<float> A) {
    using S = PlaneShape;
    constexpr int NG = S::NG, NN = S::NN, IB_W = ib_row_words(NN);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_bar[S::WARPS][3];  // geometry, node words (two stages)
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    unsigned char* geo_b = smem_raw + wp * S::WARP_B;
    uint32_t* ibs = reinterpret_cast<uint32_t*>(geo_b + S::CELLS * S::GEO_SLOT);  // [2][CELLS][IB_W]
    float* xch = reinterpret_cast<float*>(geo_b + S::CELLS * S::GEO_SLOT + 2 * S::CELLS * S::IB_B);
    uint64_t* bar = s_bar[wp];
    if (lane == 0) {
        for (int b = 0; b < 3; ++b) mbar_init(bar + b, 1);
        mbar_init_fence();
    }
    __syncwarp();
    const bool lane_ok = lane < 30;
    const int q = lane_ok ? lane / 5 : 0, i = lane_ok ? lane - 5 * q : 0;
    const int cl = q / 3, f = q - 3 * cl;
    if (A.live_end) pdl_wait();
    const int n_cell = A.live_end ? min(A.n_cell, __ldcg(A.live_end)) : A.n_cell;
    const int split = A.nfld / A.nfld_item;
    const int n_item = (n_cell + S::CELLS - 1) / S::CELLS * split;
    const int step = gridDim.x * S::WARPS;
    const int first = blockIdx.x * S::WARPS + wp;
    const size_t row_u = (size_t)(A.nfld / 3) * (S::CHUNK_W / 3);
    const float* geo = reinterpret_cast<const float*>(geo_b + cl * S::GEO_SLOT) + i * 25;
    float* own = xch + q * S::SQ + i * S::PI;   // + c*SC + p
    float* line = xch + q * S::SQ + 5 * i;      // + c*SC + s*PI + k

    auto copy_geo = [&](int item) {
        if (lane != 0) return;
        const int e0 = item / split * S::CELLS, nc = min(S::CELLS, n_cell - e0);
        fence_proxy_async_smem();
        mbar_expect_tx(bar, (unsigned)(nc * S::GEO_B));
        for (int c = 0; c < nc; ++c)
            bulk_copy_g2s(geo_b + c * S::GEO_SLOT, A.geom + (size_t)(e0 + c) * geo_row<float>(NN), S::GEO_B, bar);
    };
    auto copy_words = [&](int item, int st) {
        if (lane != 0) return;
        const int e0 = item / split * S::CELLS, nc = min(S::CELLS, n_cell - e0);
        fence_proxy_async_smem();
        mbar_expect_tx(bar + 1 + st, (unsigned)(nc * S::IB_B));
        bulk_copy_g2s(ibs + st * S::CELLS * IB_W, A.ibool_padded + (size_t)e0 * IB_W, (unsigned)(nc * S::IB_B), bar + 1 + st);
    };
    // a wait that gave up: flag it, give the copies in flight a second
    // bounded wait, leave (the whole warp)
    auto give_up = [&](unsigned pg, int b1, unsigned p1, int b2, unsigned p2) {
        if (lane == 0) {
            atomicOr(A.err, 1u);
            mbar_wait(bar, pg);
            if (b1 >= 0) mbar_wait(bar + b1, p1);
            if (b2 >= 0) mbar_wait(bar + b2, p2);
            bulk_wait_all();
        }
    };

    if (first < n_item) {
        copy_words(first, 0);
        copy_geo(first);
    }
    pdl_wait();
    pdl_launch();
    int it = 0;
    for (int item = first; item < n_item; item += step, ++it) {
        const int st = it & 1, next = item + step;
        const unsigned pw = (unsigned)(it >> 1) & 1u, pg = (unsigned)it & 1u;
        if (next < n_item) copy_words(next, st ^ 1);
        if (__any_sync(0xffffffffu, !mbar_wait(bar + 1 + st, pw))) {
            give_up(pg, 1 + st, pw, next < n_item ? 2 - st : -1, (unsigned)((it + 1) >> 1) & 1u);
            return;
        }
        const int e0 = item / split * S::CELLS, e = e0 + cl;
        const bool in = lane_ok && e < n_cell;
        const uint32_t* words = ibs + (st * S::CELLS + cl) * IB_W;
        const int mdl = A.multi && in ? (int)words[NN] : 0;
        const int src0 = in && A.src_head ? __ldg(A.src_head + e) : -1;
        const int d0 = item % split * A.nfld_item, d1 = d0 + A.nfld_item;
        for (int g0 = d0; g0 < d1; g0 += 3) {
            // row j of component c: points k = 0, 1 | 2, 3 | 4
            float2 u2[3][NG][2];
            float u1[3][NG];
#pragma unroll
            for (int j = 0; j < NG; ++j) {
                float4 t[NG];
#pragma unroll
                for (int k = 0; k < NG; ++k) {
                    const uint32_t w = in ? words[i * 25 + j * NG + k] & kNodeMask : 0u;
                    t[k] = reinterpret_cast<const float4*>(A.ut)[(size_t)w * A.nfld + g0 + f];
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    u2[0][j][h] = make_float2(t[2 * h].x, t[2 * h + 1].x);
                    u2[1][j][h] = make_float2(t[2 * h].y, t[2 * h + 1].y);
                    u2[2][j][h] = make_float2(t[2 * h].z, t[2 * h + 1].z);
                }
                u1[0][j] = t[4].x, u1[1][j] = t[4].y, u1[2][j] = t[4].z;
            }
            auto u_at = [&](int c, int j, int k) -> float {
                return k == 4 ? u1[c][j] : (k & 1 ? u2[c][j][k / 2].y : u2[c][j][k / 2].x);
            };
            if (lane == 0) bulk_wait_read();  // the contributions before have left the exchange array
            __syncwarp();
            if (lane_ok) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int p = 0; p < 25; ++p) own[c * S::SC + p] = u_at(c, p / NG, p % NG);
            }
            __syncwarp();
            // the xi contractions along this lane's five lines, in place
            auto contract = [&](auto coef) {
#pragma unroll 1  // a third of the code: instruction fetch shows here
                for (int c = 0; c < 3; ++c) {
                    auto lines = [&](auto zero, int k) {
                        decltype(zero) v[NG];
                        float* l = line + c * S::SC + k;
#pragma unroll
                        for (int t = 0; t < NG; ++t) vload(l + t * S::PI, 1, v[t]);
#pragma unroll
                        for (int s = 0; s < NG; ++s) {
                            decltype(zero) x = vmul(coef(zero, s, 0), v[0]);
#pragma unroll
                            for (int t = 1; t < NG; ++t) x = vfma(coef(zero, s, t), v[t], x);
                            vstore(l + s * S::PI, 1, x);
                        }
                    };
                    lines(float2{}, 0);
                    lines(float2{}, 2);
                    lines(0.f, 4);
                }
            };
            struct Coef {
                const GatherArgs<float>& A;
                __device__ __forceinline__ float2 operator()(float2, int a, int b) const { return A.D2[a * 5 + b]; }
                __device__ __forceinline__ float operator()(float, int a, int b) const { return A.D[a * 5 + b]; }
            };
            const Coef D{A};
            if (lane_ok) contract([&](auto z, int s, int t) { return D(z, s, t); });
            if (g0 == d0 && __any_sync(0xffffffffu, !mbar_wait(bar, pg))) {
                give_up(pg, next < n_item ? 2 - st : -1, (unsigned)((it + 1) >> 1) & 1u, -1, 0);
                return;
            }
            __syncwarp();
            float2 r2[3][NG][2];
            float r1[3][NG];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int j = 0; j < NG; ++j) {
                    r2[c][j][0] = r2[c][j][1] = make_float2(0.f, 0.f);
                    r1[c][j] = 0.f;
                }
            if (lane_ok) {
#pragma unroll
                for (int j = 0; j < NG; ++j) {
                    float z[3][NG];  // the zeta fluxes of the row
                    // d/d-zeta at k: a scalar contraction along the row
                    auto dz = [&](int c, int k) -> float {
                        float x = A.D[k * NG] * u_at(c, j, 0);
#pragma unroll
                        for (int s = 1; s < NG; ++s) x = vfma(A.D[k * NG + s], u_at(c, j, s), x);
                        return x;
                    };
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k = 2 * h, p = j * NG + k;
                        float2 g[3][3], fl[3][3];
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            vload(own + c * S::SC + p, 1, g[c][0]);
                            g[c][1] = vmul(A.D2[j * NG], u2[c][0][h]);
#pragma unroll
                            for (int s = 1; s < NG; ++s) g[c][1] = vfma(A.D2[j * NG + s], u2[c][s][h], g[c][1]);
                            g[c][2] = make_float2(dz(c, k), dz(c, k + 1));
                        }
                        point_fluxes<OFF>(geo + p, NN, 1, g, fl);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            vstore(own + c * S::SC + p, 1, fl[0][c]);
#pragma unroll
                            for (int s = 0; s < NG; ++s) r2[c][s][h] = vfma(A.D2[j * NG + s], fl[1][c], r2[c][s][h]);
                            z[c][k] = fl[2][c].x;
                            z[c][k + 1] = fl[2][c].y;
                        }
                    }
                    {
                        const int p = j * NG + 4;
                        float g[3][3], fl[3][3];
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            g[c][0] = own[c * S::SC + p];
                            g[c][1] = A.D[j * NG] * u1[c][0];
#pragma unroll
                            for (int s = 1; s < NG; ++s) g[c][1] = vfma(A.D[j * NG + s], u1[c][s], g[c][1]);
                            g[c][2] = dz(c, 4);
                        }
                        point_fluxes<OFF>(geo + p, NN, 1, g, fl);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            own[c * S::SC + p] = fl[0][c];
#pragma unroll
                            for (int s = 0; s < NG; ++s) r1[c][s] = vfma(A.D[j * NG + s], fl[1][c], r1[c][s]);
                            z[c][4] = fl[2][c];
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int k = 0; k < NG; ++k) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                r2[c][j][h].x = vfma(A.D[k * NG + 2 * h], z[c][k], r2[c][j][h].x);
                                r2[c][j][h].y = vfma(A.D[k * NG + 2 * h + 1], z[c][k], r2[c][j][h].y);
                            }
                            r1[c][j] = vfma(A.D[k * NG + 4], z[c][k], r1[c][j]);
                        }
                }
            }
            __syncwarp();  // and the geometry has been read
            if (g0 + 3 >= d1 && next < n_item) copy_geo(next);
            if (lane_ok) contract([&](auto z, int s, int t) { return D(z, t, s); });
            __syncwarp();
            float r[3][25];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int j = 0; j < NG; ++j)
#pragma unroll
                    for (int k = 0; k < NG; ++k) {
                        const float x = k == 4 ? r1[c][j] : (k & 1 ? r2[c][j][k / 2].y : r2[c][j][k / 2].x);
                        r[c][j * NG + k] = -(x + own[c * S::SC + j * NG + k]);
                    }
            // point force (solver.cpp:577-605)
            if (src0 >= 0 && A.mstf) {
                const int d = g0 + f, fs = A.fset[d], dir = A.dir[d];
                const float stf = __ldcg(A.mstf + mdl * A.n_set + fs);
                for (int sl = stf != 0.f ? src0 : -1; sl >= 0; sl = __ldg(A.src_next + sl)) {
                    if (A.src_set && __ldg(A.src_set + sl) != fs) continue;
#pragma unroll
                    for (int p = 0; p < 25; ++p) {
                        const float sw = stf * __ldg(A.src_w + (size_t)sl * NN + i * 25 + p);
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            if (c == dir) r[c][p] += sw;
                    }
                }
            }
            __syncwarp();  // every lane has read the exchange array
            if (lane_ok) {
                float* out = xch + cl * S::CHUNK_W + i * 225 + 3 * f;
#pragma unroll
                for (int p = 0; p < 25; ++p)
#pragma unroll
                    for (int c = 0; c < 3; ++c) out[p * 9 + c] = r[c][p];
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                const int nc = min(S::CELLS, n_cell - e0);
                for (int c = 0; c < nc; ++c)
                    bulk_copy_s2g(A.contrib + ((size_t)(e0 + c) * row_u + (size_t)(g0 / 3) * (S::CHUNK_W / 3)) * 3,
                                  xch + c * S::CHUNK_W, (unsigned)(S::CHUNK_W * 4));
                bulk_commit();
            }
        }
    }
    if (lane == 0) bulk_wait_all();
}

// Predictor only (start of a run or after a state overwrite).
// Nodes g >= hv_begin hold the half-step velocity (v + dt/2 a) in w32.
template <typename Real>
__global__ void predict_kernel(long long n_node, int F, const double* u, const double* v, const Real* a,
                               Real* ut, double dt, double half_dt2, const uint8_t* node_model,
                               const ModelConst* mc, long long hv_begin, const float* w32) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long total = n_node * F;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const long long g = idx / F;
        const int f = (int)(idx - g * F);
        double h = dt, h2 = half_dt2;
        if (node_model) {
            const ModelConst& K = mc[node_model[g]];
            h = K.dt;
            h2 = K.half_dt2;
        }
        ut[padded_index(g, f, F)] =
            g >= hv_begin ? (Real)(u[idx] + h * (double)w32[idx]) : (Real)(u[idx] + h * v[idx] + h2 * (double)a[idx]);
        if (f % 3 == 2) ut[padded_index(g, f, F) + 1] = Real(0);
    }
}

template <typename Real, typename Out>
struct RecArgs {
    int n_rec;
    const int* rec_cell;    // [n_rec] device cell index
    const uint32_t* ibool;
    const Real* geom;
    const Real* dmat;
    const double* u;        // [node][3*n_field]
    const double* v;
    const Real* a;
    long long n_node;
    Out* out;               // [NFLD] of strain [n_rec][NN][6], u, v, a [n_rec][NN][3]
    // nodes g >= hv_begin hold the half-step velocity w (w32): a = f/m from
    // the step's assembled force, v = w - dt/2 a
    long long hv_begin;
    const float* w32;
    const Real* force;      // [node][NFLD][4]
    const Real* inv_mass;   // [node]
    const uint8_t* node_model;
    const ModelConst* mc;
    double dt;
};

// Snapshot of the recording cells: strain from the gathered corrected
// displacement (solver.cpp:282-335) plus u, v, a at every cell node
// (solver.cpp:485-504).  One block per recording cell.
template <typename Real, int NG, int NFLD, typename Out>
__global__ void record_kernel(RecArgs<Real, Out> A) {
    using S = Shape<NG>;
    constexpr int NN = S::NN, F = 3 * NFLD;
    __shared__ double su[F][NN];
    __shared__ double sD[NG * NG];
    const int ci = blockIdx.x;
    const int p = threadIdx.x;
    if (p < NG * NG) sD[p] = (double)A.dmat[p];
    const int e = A.rec_cell[ci];
    uint32_t g = 0;
    if (p < NN) {
        g = A.ibool[(size_t)e * NN + p] & kNodeMask;
        for (int f = 0; f < F; ++f) su[f][p] = A.u[(size_t)g * F + f];
    }
    __syncthreads();
    if (p >= NN) return;
    const int i = p / (NG * NG), j = (p / NG) % NG, k = p % NG;
    double dd[9];
    const Real* gp = A.geom + (size_t)e * geo_row<Real>(NN) + p;
    for (int q = 0; q < 9; ++q) dd[q] = (double)gp[q * NN];
    for (int d = 0; d < NFLD; ++d) {
        double gx[3] = {0, 0, 0}, gy[3] = {0, 0, 0}, gz[3] = {0, 0, 0};
        for (int s = 0; s < NG; ++s) {
            const double Di = sD[i * NG + s], Dj = sD[j * NG + s], Dk = sD[k * NG + s];
            for (int c = 0; c < 3; ++c) {
                gx[c] += Di * su[d * 3 + c][(s * NG + j) * NG + k];
                gy[c] += Dj * su[d * 3 + c][(i * NG + s) * NG + k];
                gz[c] += Dk * su[d * 3 + c][(i * NG + j) * NG + s];
            }
        }
        double gr[3][3];
        for (int c = 0; c < 3; ++c) {
            gr[c][0] = gx[c] * dd[0] + gy[c] * dd[1] + gz[c] * dd[2];
            gr[c][1] = gx[c] * dd[3] + gy[c] * dd[4] + gz[c] * dd[5];
            gr[c][2] = gx[c] * dd[6] + gy[c] * dd[7] + gz[c] * dd[8];
        }
        const size_t points = (size_t)A.n_rec * NN, q = (size_t)ci * NN + p;
        Out* o = A.out + (size_t)d * points * 15 + q * 6;
        Out* ou = A.out + ((size_t)d * 15 + 6) * points + q * 3;
        Out *ov = ou + 3 * points, *oa = ov + 3 * points;
        o[0] = (Out)gr[0][0];
        o[1] = (Out)gr[1][1];
        o[2] = (Out)gr[2][2];
        o[3] = (Out)(0.5 * (gr[0][1] + gr[1][0]));
        o[4] = (Out)(0.5 * (gr[0][2] + gr[2][0]));
        o[5] = (Out)(0.5 * (gr[1][2] + gr[2][1]));
        if ((long long)g >= A.hv_begin) {
            const double h = A.node_model ? A.mc[A.node_model[g]].dt : A.dt;
            const Real im = A.inv_mass[g];
            for (int c = 0; c < 3; ++c) {
                const double an = (double)(Real)(A.force[((size_t)g * NFLD + d) * 4 + c] * im);
                ou[c] = (Out)A.u[(size_t)g * F + d * 3 + c];
                ov[c] = (Out)((double)A.w32[(size_t)g * F + d * 3 + c] - 0.5 * h * an);
                oa[c] = (Out)an;
            }
        } else {
            for (int c = 0; c < 3; ++c) {
                ou[c] = (Out)A.u[(size_t)g * F + d * 3 + c];
                ov[c] = (Out)A.v[(size_t)g * F + d * 3 + c];
                oa[c] = (Out)A.a[(size_t)g * F + d * 3 + c];
            }
        }
    }
}


// Half-step velocity state (w32) <-> (v, a) at the nodes g >= hv_begin.
// to_full: v_out = w - dt/2 a, a_out = a with a = f/m from the assembled
// force (a_from_force) or the stored a (state set since the last step);
// otherwise (from_full): w = v + dt/2 a.  One thread per (node, value).
template <typename Real>
__global__ void half_v_kernel(long long n_node, int F, long long hv_begin, bool to_full, bool a_from_force,
                              const double* v, float* w32, const Real* a, const Real* force, const Real* inv_mass,
                              const uint8_t* node_model, const ModelConst* mc, double dt, double* v_out,
                              Real* a_out) {
    const long long total = (n_node - hv_begin) * F;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long g = hv_begin + t / F;
        const int f = (int)(t % F);
        const size_t i = (size_t)g * F + f;
        const double h = node_model ? mc[node_model[g]].dt : dt;
        if (to_full) {
            const double an = a_from_force ? (double)(Real)(force[padded_index(g, f, F)] * inv_mass[g]) : (double)a[i];
            v_out[i] = (double)w32[i] - 0.5 * h * an;
            a_out[i] = (Real)an;
        } else {
            w32[i] = (float)(v[i] + 0.5 * h * (double)a[i]);
        }
    }
}

// u, v or a of wavefield `field` at the nodes [n0, n1) of the mesh's order,
// out[node - n0][3] as double: one thread per value, the scattered side the read.
// inv: node -> device node (nullptr: device nodes [n0, n1)).  what: 0 u, 1 v, 2 a; nodes >= hv_begin
// hold the half-step velocity, as in half_v_kernel.
template <typename Real>
__global__ void state_kernel(long long n0, long long n1, int F, int field, int what, const int* inv, const double* u,
                             const double* v, const Real* a, long long hv_begin, bool a_from_force, const float* w32,
                             const Real* force, const Real* inv_mass, const uint8_t* node_model, const ModelConst* mc,
                             double dt, double* out) {
    const long long total = (n1 - n0) * 3;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long n = t / 3;
        const int f = field * 3 + (int)(t - n * 3);
        const long long g = inv ? inv[n0 + n] : n0 + n;
        const size_t i = (size_t)g * F + f;
        double x;
        if (what == 0) {
            x = u[i];
        } else if (g < hv_begin) {
            x = what == 1 ? v[i] : (double)a[i];
        } else {
            const double h = node_model ? mc[node_model[g]].dt : dt;
            const double an = a_from_force ? (double)(Real)(force[padded_index(g, f, F)] * inv_mass[g]) : (double)a[i];
            x = what == 1 ? (double)w32[i] - 0.5 * h * an : (double)(Real)an;
        }
        out[t] = x;
    }
}

// Recording nodes merged across the recording cells that share them (the
// strain Green's-function extraction of postprocess/cpp/main.cpp:300-425):
// strain mass-weighted, sum(m_p e_p) / sum(m_p) over the node's (cell, point)
// occurrences; u, v, a averaged.  One thread per (wavefield, node, value),
// reading the snapshot's cell-point records (RecArgs::out, per_field points)
// and writing merged[field][node][15] behind them in the same slot.
template <typename Out>
__global__ void merge_nodes_kernel(int n_field, int n_unique, long long per_field, const int* ptr, const int* occ,
                                   const double* w, Out* slot) {
    const long long total = (long long)n_field * n_unique * 15;
    Out* merged = slot + (size_t)n_field * per_field * 15;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(t % 15);
        const long long fn = t / 15;
        const int node = (int)(fn % n_unique), f = (int)(fn / n_unique);
        // component c of the field's points, `w0` values apart
        const int w0 = c < 6 ? 6 : 3;
        const Out* src = slot + (size_t)f * per_field * 15 + (c < 6 ? c : per_field * (c / 3 * 3) + c % 3);
        double acc = 0.0, ws = 0.0;
        for (int k = ptr[node]; k < ptr[node + 1]; ++k) {
            const double wk = c < 6 ? w[k] : 1.0;
            acc += wk * (double)src[(size_t)occ[k] * w0];
            ws += wk;
        }
        merged[((size_t)f * n_unique + node) * 15 + c] = (Out)(ws > 0.0 ? acc / ws : 0.0);
    }
}

}  // namespace gfb
