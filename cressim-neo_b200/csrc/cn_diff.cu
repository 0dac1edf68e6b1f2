// cn_diff.cu -- differentiable XPBD rollout: forward substeps with checkpoints and a hand-written
// adjoint (no reference counterpart: the reference has no gradients).
//
// The rollout is the soft-body substep of the particle path -- predict, `iterations` Jacobi
// iterations of edge-distance then tet-volume constraints (solve writes per-constraint correction
// records, apply gathers them per particle in ascending constraint order), velocity update --
// with pinned particles and no contacts.  The forward math below follows the product kernels
// (k_predictKeys, k_solveEdges, k_applyPair, k_solveTets, k_applyQuad, k_updateVelocities)
// expression for expression, so in float it reproduces their bits.
//
// The adjoint runs the iterations backwards: per constraint, the vector-Jacobian product of
// (corrections, lambda') with respect to (positions, lambda, compliance) is written out in reverse
// (edgeAdjoint, tetAdjoint; about twice the forward's operations, where tangents of every input
// would take 7 and 14 times as many), and goes to records that each particle gathers in ascending
// constraint order (deterministic, no atomics).  Positions and velocities are checkpointed at the start of every
// `checkpoint_interval`-th substep; backward recomputes one segment of substeps from its
// checkpoint, then one substep's iteration states at a time.  A substep and a substep's adjoint are
// each one CUDA graph, captured at first use (the launches of 8 substeps x 20 iterations took the host
// longer than the device).  47,385 tets, 8 substeps x 20 iterations, forward and backward: 25.96 -> 9.41 ms
// against dual numbers, copied states and single launches, the same error against 64 bits.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/cn_physics.h"
#include "cn_internal.h"

using cn::setError;

namespace {

constexpr int kDiffThreads = 256;
inline unsigned gridOf(size_t n) { return n == 0 ? 1u : unsigned((n + kDiffThreads - 1) / kDiffThreads); }

// ---------------------------------------------------------------- vectors
__device__ __forceinline__ float sqrtD(float a) { return sqrtf(a); }
__device__ __forceinline__ double sqrtD(double a) { return sqrt(a); }
__device__ __forceinline__ float absD(float a) { return fabsf(a); }
__device__ __forceinline__ double absD(double a) { return fabs(a); }

template <class S> struct V3 {
    S x, y, z;
};
template <class S> __device__ __forceinline__ V3<S> operator+(const V3<S> &a, const V3<S> &b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class S> __device__ __forceinline__ V3<S> operator-(const V3<S> &a, const V3<S> &b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class S> __device__ __forceinline__ V3<S> operator-(const V3<S> &a) { return {-a.x, -a.y, -a.z}; }
template <class S> __device__ __forceinline__ V3<S> operator*(const V3<S> &a, const S &s) { return {a.x * s, a.y * s, a.z * s}; }
template <class S> __device__ __forceinline__ V3<S> operator*(const S &s, const V3<S> &a) { return {s * a.x, s * a.y, s * a.z}; }
template <class S> __device__ __forceinline__ V3<S> operator/(const V3<S> &a, const S &s) { return {a.x / s, a.y / s, a.z / s}; }
template <class S> __device__ __forceinline__ S dot3(const V3<S> &a, const V3<S> &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <class S> __device__ __forceinline__ V3<S> cross3(const V3<S> &a, const V3<S> &b)
{
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

template <class T> struct P4 {
    T x, y, z, w;
};

// ---------------------------------------------------------------- constraint math
// physics_soft_solve_edge_constraints.cs.hlsl:10-74 (k_solveEdges): what the forward and the adjoint share.
// False when the record is written as zeros (no mass, zero length, no denominator): then lambda' = lambda.
template <class T> struct EdgeTerms {
    V3<T> delta;
    T len, alpha, den, dl;
};
template <class T>
__device__ __forceinline__ bool edgeTerms(const V3<T> &a, const V3<T> &b, T wA, T wB, T rest, T compliance, T lambda, T dt,
                                          EdgeTerms<T> &e)
{
    const T eps = T(1.0e-6);
    const T wSum = wA + wB;
    e.delta = b - a;
    const T l2 = dot3(e.delta, e.delta);
    if (!(wSum > eps && l2 > eps)) return false;
    e.len = sqrtD(l2);
    const T dt2 = dt * dt;
    e.alpha = compliance / (dt2 > eps ? dt2 : eps); // max(compliance, 0): compliance > 0 here
    const T Cv = e.len - rest;
    e.den = wSum + e.alpha;
    if (!(e.den > eps)) return false;
    e.dl = -(Cv + e.alpha * lambda) / e.den;
    return true;
}

template <class T>
__device__ __forceinline__ bool edgeProject(const V3<T> &a, const V3<T> &b, T wA, T wB, T rest, T compliance, T lambda, T dt,
                                            T relax, V3<T> &cA, V3<T> &cB, T &lambdaOut)
{
    EdgeTerms<T> e;
    lambdaOut = lambda;
    if (!edgeTerms(a, b, wA, wB, rest, compliance, lambda, dt, e)) return false;
    const V3<T> gA = (-e.delta) / e.len;
    const V3<T> gB = -gA;
    lambdaOut = lambda + e.dl;
    cA = ((wA * e.dl) * gA) * relax;
    cB = ((wB * e.dl) * gB) * relax;
    return true;
}

// Adjoints of b (that of a is its negative) and lambda from those of the corrections and of lambda'.
// With u = delta / len: cA = -wA relax dl u, cB = wB relax dl u.
template <class T>
__device__ __forceinline__ V3<T> edgeAdjoint(const EdgeTerms<T> &e, T wA, T wB, T relax, const V3<T> &gA, const V3<T> &gB, T gL,
                                             T &gLambda)
{
    const V3<T> u = e.delta / e.len;
    const V3<T> m = (gB * (wB * relax)) - (gA * (wA * relax));
    const T D = gL + dot3(m, u);          // of dl
    const V3<T> U = m * e.dl;             // of u
    gLambda = gL - D * (e.alpha / e.den);
    return (u * (-D / e.den)) + ((U - (u * dot3(U, u))) / e.len);
}

// physics_soft_solve_tet_constraints.cs.hlsl:15-87 (k_solveTets).  False when the reference keeps the
// previous record (no mass, no denominator).
template <class T> struct TetTerms {
    V3<T> e1, e2, e3; // p1 - p0, p2 - p0, p3 - p0
    V3<T> a, b;       // p3 - p1, p2 - p1
    V3<T> g[4];
    T k6, alpha, den, dl;
};
template <class T>
__device__ __forceinline__ bool tetTerms(const V3<T> p[4], const T w[4], T rest, T compliance, T lambda, T dt, TetTerms<T> &t)
{
    const T eps = T(1.0e-6);
    if ((w[0] + w[1] + w[2] + w[3]) <= eps) return false;
    t.e1 = p[1] - p[0];
    t.e2 = p[2] - p[0];
    t.e3 = p[3] - p[0];
    t.a = p[3] - p[1];
    t.b = p[2] - p[1];
    const T sv = dot3(cross3(t.e1, t.e2), t.e3) / T(6);
    const T vs = sv >= T(0) ? T(1) : T(-1);
    const T Cv = absD(sv) - (rest > T(0) ? rest : T(0));
    t.k6 = vs / T(6);
    t.g[0] = cross3(t.a, t.b) * t.k6;
    t.g[1] = cross3(t.e2, t.e3) * t.k6;
    t.g[2] = cross3(t.e3, t.e1) * t.k6;
    t.g[3] = cross3(t.e1, t.e2) * t.k6;
    const T sg = w[0] * dot3(t.g[0], t.g[0]) + w[1] * dot3(t.g[1], t.g[1]) + w[2] * dot3(t.g[2], t.g[2]) +
                 w[3] * dot3(t.g[3], t.g[3]);
    const T dt2 = dt * dt;
    t.alpha = compliance / (dt2 > eps ? dt2 : eps);
    t.den = sg + t.alpha;
    if (!(t.den > eps)) return false;
    t.dl = -(Cv + t.alpha * lambda) / t.den;
    return true;
}

// Adjoints of the four positions, lambda and the scaled compliance from those of the corrections (gC) and
// of lambda'.  With out_j = w_j relax dl g_j and dl = -(C + alpha lambda) / den, den = sum w_j |g_j|^2 + alpha;
// the gradients are cross products, whose adjoints are cross products, and dC / dp_j = g_j.
template <class T>
__device__ __forceinline__ void tetAdjoint(const TetTerms<T> &t, const T w[4], T relax, const V3<T> gC[4], T lambda, T gL,
                                           V3<T> gP[4], T &gLambda, T &gAlpha)
{
    T D = gL;
#pragma unroll
    for (int j = 0; j < 4; ++j) D += (w[j] * relax) * dot3(gC[j], t.g[j]);
    const T inv = T(1) / t.den;
    const T S = -(D * t.dl) * inv; // of den
    const T V = -D * inv;          // of C
    gLambda = gL + V * t.alpha;
    gAlpha = V * lambda + S;
    V3<T> h[4];                    // of k6 x the cross products
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = ((gC[j] * (w[j] * relax * t.dl)) + (t.g[j] * (T(2) * w[j] * S))) * t.k6;
    const V3<T> gE1 = cross3(h[2], t.e3) + cross3(t.e2, h[3]);
    const V3<T> gE2 = cross3(t.e3, h[1]) + cross3(h[3], t.e1);
    const V3<T> gE3 = cross3(h[1], t.e2) + cross3(t.e1, h[2]);
    const V3<T> ga = cross3(t.b, h[0]), gb = cross3(h[0], t.a);
    gP[0] = (t.g[0] * V) - (gE1 + gE2 + gE3);
    gP[1] = (t.g[1] * V) + (gE1 - (ga + gb));
    gP[2] = (t.g[2] * V) + (gE2 + gb);
    gP[3] = (t.g[3] * V) + (gE3 + ga);
}

// ---------------------------------------------------------------- device scene
template <class T> struct DScene {
    uint32_t N = 0, E = 0, T_ = 0;
    const T *w = nullptr;          // inverse mass
    const T *damp = nullptr;       // per-particle velocity damping (contact material .z)
    const uint2 *edgePair = nullptr;
    const T *edgeRest = nullptr, *edgeCompliance = nullptr;
    const uint32_t *edgeEnabled = nullptr;
    const uint4 *tetIdx = nullptr;
    const T *tetRest = nullptr;
    // per particle its records (first, count), per constraint entry the record it writes (kNone: none)
    const uint2 *edgeRanges = nullptr, *tetRanges = nullptr;
    const uint2 *edgeDst = nullptr;
    const uint4 *tetDst = nullptr;
    T g[3] = {T(0), T(0), T(0)};
    T relax = T(0.2);
};

template <class T> __device__ __forceinline__ V3<T> xyzOf(const P4<T> &p) { return {p.x, p.y, p.z}; }

constexpr uint32_t kNone = 0xffffffffu;
template <class T> __device__ __forceinline__ void putRecord(P4<T> *records, uint32_t at, const V3<T> &v)
{
    if (at != kNone) records[at] = {v.x, v.y, v.z, T(0)};
}

// k_predictKeys for a solid particle (gravity scale 1): the predicted positions go to xOut
template <class T> __global__ void k_dPredict(DScene<T> s, const P4<T> *x, P4<T> *xOut, P4<T> *v, P4<T> *xprev, T dt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.N) return;
    const P4<T> p = x[i];
    xprev[i] = {p.x, p.y, p.z, T(0)};
    if (s.w[i] <= T(1.0e-6)) {
        v[i] = {T(0), T(0), T(0), T(0)};
        xOut[i] = p;
        return;
    }
    const P4<T> vv = v[i];
    const T gs = dt * T(1);
    const V3<T> vel = V3<T>{vv.x, vv.y, vv.z} + V3<T>{s.g[0], s.g[1], s.g[2]} * gs;
    const V3<T> pp = V3<T>{p.x, p.y, p.z} + vel * dt;
    v[i] = {vel.x, vel.y, vel.z, T(0)};
    xOut[i] = {pp.x, pp.y, pp.z, p.w};
}

// The iteration kernels are launched with programmatic stream serialization: what their predecessor does
// not write loads ahead of the wait (as in the solver's kernels: cn::pdlEnter).
template <class T>
__global__ void __launch_bounds__(kDiffThreads) k_dEdges(DScene<T> s, const P4<T> *x, const T *lambdaIn, T *lambdaOut, P4<T> *corr,
                                                         T dt, bool first)
{
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    uint2 ab = make_uint2(0u, 0u), d = make_uint2(kNone, kNone);
    T wA = T(0), wB = T(0), rest = T(0), comp = T(0), lambda = T(0);
    bool enabled = false;
    if (e < s.E) {
        ab = s.edgePair[e];
        d = s.edgeDst[e];
        wA = s.w[ab.x];
        wB = s.w[ab.y];
        rest = s.edgeRest[e];
        comp = s.edgeCompliance[e] > T(0) ? s.edgeCompliance[e] : T(0);
        if (!first) lambda = lambdaIn[e];
        enabled = s.edgeEnabled[e] != 0u;
    }
    cn::pdlEnter();
    if (e >= s.E) return;
    V3<T> cA{T(0), T(0), T(0)}, cB = cA;
    T lo = lambda;
    if (enabled) edgeProject<T>(xyzOf(x[ab.x]), xyzOf(x[ab.y]), wA, wB, rest, comp, lambda, dt, s.relax, cA, cB, lo);
    lambdaOut[e] = lo;
    putRecord(corr, d.x, cA);
    putRecord(corr, d.y, cB);
}

template <class T>
__global__ void __launch_bounds__(kDiffThreads) k_dTets(DScene<T> s, const P4<T> *x, const T *compliance, const T *lambdaIn,
                                                        T *lambdaOut, P4<T> *corr, T dt, bool first)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint4 q = make_uint4(0u, 0u, 0u, 0u), d = make_uint4(kNone, kNone, kNone, kNone);
    T w[4] = {T(0), T(0), T(0), T(0)}, rest = T(0), comp = T(0), lambda = T(0);
    if (t < s.T_) {
        q = s.tetIdx[t];
        d = s.tetDst[t];
        w[0] = s.w[q.x];
        w[1] = s.w[q.y];
        w[2] = s.w[q.z];
        w[3] = s.w[q.w];
        rest = s.tetRest[t];
        comp = compliance[t] > T(0) ? compliance[t] : T(0);
        if (!first) lambda = lambdaIn[t];
    }
    cn::pdlEnter();
    if (t >= s.T_) return;
    const V3<T> p[4] = {xyzOf(x[q.x]), xyzOf(x[q.y]), xyzOf(x[q.z]), xyzOf(x[q.w])};
    TetTerms<T> m;
    if (!tetTerms<T>(p, w, rest, comp, lambda, dt, m)) { // the previous record stays (the reference's behaviour)
        lambdaOut[t] = lambda;
        return;
    }
    lambdaOut[t] = lambda + m.dl;
    const uint32_t dst[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) putRecord(corr, dst[k], ((w[k] * m.dl) * m.g[k]) * s.relax);
}

// out[i] = in[i] + the sum of i's records in ascending constraint order: the apply of a family (k_applyGather;
// particles without mass keep their position), and of the adjoint records (kAdjoint: every particle).
// Four lanes per particle, one per component, sixteen records in flight.  In place when out == in.
constexpr uint32_t kLanes = 4u, kAhead = 16u;
template <class T, bool kAdjoint>
__global__ void __launch_bounds__(kDiffThreads) k_dGather(DScene<T> s, const P4<T> *in, P4<T> *out, const uint2 *ranges,
                                                          const P4<T> *records)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x, i = q / kLanes, comp = q % kLanes;
    const bool live = i < s.N;
    T x = T(0);
    bool moves = false;
    uint2 r = make_uint2(0u, 0u);
    if (live) {
        x = reinterpret_cast<const T *>(in)[q]; // not written by the solve this kernel follows
        r = ranges[i];
        moves = comp < 3u && (kAdjoint || s.w[i] > T(1.0e-6));
    }
    cn::pdlEnter();
    if (!live) return;
    if (moves) {
        const T *src = reinterpret_cast<const T *>(records + r.x) + comp;
        T total = kAdjoint ? x : T(0);
        for (uint32_t k = 0; k < r.y; k += kAhead) {
            T c[kAhead];
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j)
                if (k + j < r.y) c[j] = src[kLanes * (k + j)];
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j)
                if (k + j < r.y) total += c[j];
        }
        x = kAdjoint ? total : x + total;
    }
    if (moves || out != in) reinterpret_cast<T *>(out)[q] = kAdjoint && comp == 3u ? T(0) : x;
}

// k_updateVelocities for a solid particle
template <class T> __global__ void k_dVelocity(DScene<T> s, const P4<T> *x, const P4<T> *xprev, P4<T> *v, T dt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.N) return;
    if (s.w[i] <= T(1.0e-6) || dt <= T(1.0e-6)) {
        v[i] = {T(0), T(0), T(0), T(0)};
        return;
    }
    const T d = s.damp[i] > T(0) ? s.damp[i] : T(0);
    const T a = T(1) - d * dt;
    const T ds = a > T(0) ? a : T(0);
    const V3<T> vel = ((xyzOf(x[i]) - xyzOf(xprev[i])) / dt) * ds;
    v[i] = {vel.x, vel.y, vel.z, T(0)};
}

// ---------------------------------------------------------------- adjoint kernels
// Edge: the adjoints of a and b as records, that of the input lambda in gLambda's place.  Edge
// compliance is not a parameter here.  Corrections reach particles with mass only (the apply skips
// the rest), so the others' adjoints do not enter.
template <class T>
__global__ void __launch_bounds__(kDiffThreads) k_dEdgesBack(DScene<T> s, const P4<T> *x, const T *lambdaIn, const P4<T> *gX,
                                                             T *gLambda, P4<T> *rec, T dt)
{
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    uint2 ab = make_uint2(0u, 0u), d = make_uint2(kNone, kNone);
    T wA = T(0), wB = T(0), gl = T(0), lambda = T(0);
    V3<T> a{T(0), T(0), T(0)}, b = a;
    EdgeTerms<T> m{};
    bool wrote = false;
    if (e < s.E) { // the forward's state: recorded before the adjoint began
        ab = s.edgePair[e];
        d = s.edgeDst[e];
        wA = s.w[ab.x];
        wB = s.w[ab.y];
        gl = gLambda[e];
        lambda = lambdaIn[e];
        a = xyzOf(x[ab.x]);
        b = xyzOf(x[ab.y]);
        const T comp = s.edgeCompliance[e] > T(0) ? s.edgeCompliance[e] : T(0);
        wrote = s.edgeEnabled[e] != 0u && edgeTerms<T>(a, b, wA, wB, s.edgeRest[e], comp, lambda, dt, m);
    }
    cn::pdlEnter();
    if (e >= s.E) return;
    V3<T> gB{T(0), T(0), T(0)};
    if (wrote) {
        const V3<T> zero{T(0), T(0), T(0)};
        gB = edgeAdjoint<T>(m, wA, wB, s.relax, wA > T(1.0e-6) ? xyzOf(gX[ab.x]) : zero,
                            wB > T(1.0e-6) ? xyzOf(gX[ab.y]) : zero, gl, gl);
    }
    putRecord(rec, d.x, -gB);
    putRecord(rec, d.y, gB);
    gLambda[e] = gl;
}

// Tet: the adjoints of the four positions as records, of lambda in place, of the compliance added up.
template <class T>
__global__ void __launch_bounds__(kDiffThreads) k_dTetsBack(DScene<T> s, const P4<T> *x, const T *compliance, const T *lambdaIn,
                                                            const P4<T> *gX, T *gLambda, P4<T> *rec, T *gCompliance, T dt)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint4 q = make_uint4(0u, 0u, 0u, 0u), d = make_uint4(kNone, kNone, kNone, kNone);
    T w[4] = {T(0), T(0), T(0), T(0)}, lambda = T(0), gl = T(0), c0 = T(0);
    TetTerms<T> m{};
    bool wrote = false;
    if (t < s.T_) {
        q = s.tetIdx[t];
        d = s.tetDst[t];
        w[0] = s.w[q.x];
        w[1] = s.w[q.y];
        w[2] = s.w[q.z];
        w[3] = s.w[q.w];
        lambda = lambdaIn[t];
        gl = gLambda[t];
        c0 = compliance[t];
        const V3<T> p[4] = {xyzOf(x[q.x]), xyzOf(x[q.y]), xyzOf(x[q.z]), xyzOf(x[q.w])};
        wrote = tetTerms<T>(p, w, s.tetRest[t], c0 > T(0) ? c0 : T(0), lambda, dt, m);
    }
    cn::pdlEnter();
    if (t >= s.T_) return;
    const uint32_t id[4] = {q.x, q.y, q.z, q.w}, dst[4] = {d.x, d.y, d.z, d.w};
    V3<T> gP[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) gP[j] = {T(0), T(0), T(0)};
    if (wrote) {
        V3<T> gC[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) gC[j] = w[j] > T(1.0e-6) ? xyzOf(gX[id[j]]) : V3<T>{T(0), T(0), T(0)};
        T gAlpha;
        tetAdjoint<T>(m, w, s.relax, gC, lambda, gl, gP, gl, gAlpha);
        const T dt2 = dt * dt;
        if (c0 > T(0)) gCompliance[t] += gAlpha / (dt2 > T(1.0e-6) ? dt2 : T(1.0e-6));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) putRecord(rec, dst[j], gP[j]);
    gLambda[t] = gl;
}

// Velocity update + predict, backwards.  In: gX (adjoint of the substep's end positions),
// gV (of its end velocities), gX0 is overwritten: first with the adjoint entering the last
// iteration, later (k_dPredictBack) with the adjoint of the substep's start positions.
template <class T> __global__ void k_dVelocityBack(DScene<T> s, const P4<T> *gX, const P4<T> *gV, P4<T> *gXI, T dt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.N) return;
    P4<T> g = gX[i];
    if (s.w[i] > T(1.0e-6) && dt > T(1.0e-6)) {
        const T d = s.damp[i] > T(0) ? s.damp[i] : T(0);
        const T a = T(1) - d * dt;
        const T k = (a > T(0) ? a : T(0)) / dt;
        const P4<T> gv = gV[i];
        g.x += gv.x * k;
        g.y += gv.y * k;
        g.z += gv.z * k;
    }
    gXI[i] = g;
}

template <class T>
__global__ void k_dPredictBack(DScene<T> s, const P4<T> *gX0, const P4<T> *gV, P4<T> *gXs, P4<T> *gVs, T dt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.N) return;
    const P4<T> g0 = gX0[i];
    P4<T> gx = {g0.x, g0.y, g0.z, T(0)};
    P4<T> gv = {T(0), T(0), T(0), T(0)};
    if (s.w[i] > T(1.0e-6)) {
        if (dt > T(1.0e-6)) {
            const T d = s.damp[i] > T(0) ? s.damp[i] : T(0);
            const T a = T(1) - d * dt;
            const T k = (a > T(0) ? a : T(0)) / dt;
            const P4<T> g = gV[i];
            gx.x -= g.x * k;
            gx.y -= g.y * k;
            gx.z -= g.z * k;
        }
        gv = {g0.x * dt, g0.y * dt, g0.z * dt, T(0)};
    }
    gXs[i] = gx;
    gVs[i] = gv;
}

// ---------------------------------------------------------------- host engine
template <class T> struct Engine {
    DScene<T> s;
    uint32_t iterations = 1, substeps = 1, interval = 8;
    T dt = T(0);
    // owned device buffers
    std::vector<void *> owned;
    P4<T> *x = nullptr, *v = nullptr, *xprev = nullptr;
    T *lamE = nullptr, *lamT = nullptr;
    P4<T> *corrE = nullptr, *corrT = nullptr;
    P4<T> *ckX = nullptr, *ckV = nullptr;     // checkpoints: (substeps / interval + 1) x N
    P4<T> *segX = nullptr, *segV = nullptr;   // one segment's substep starts: interval x N
    P4<T> *itX0 = nullptr, *itX1 = nullptr;   // one substep's iteration states: iterations x N
    T *itLE = nullptr, *itLT = nullptr;       // iterations x E, iterations x T
    P4<T> *gX = nullptr, *gV = nullptr, *gA = nullptr, *gB = nullptr;
    T *gLE = nullptr, *gLT = nullptr;
    P4<T> *recE = nullptr, *recT = nullptr;
    T *compliance = nullptr, *gCompliance = nullptr; // the forward's tet compliances, their adjoint
    bool forwardDone = false;
    // one substep, and one substep with its iteration states and its adjoint, on the buffers above
    cudaGraphExec_t stepGraph = nullptr, adjointGraph = nullptr;

    template <class U> U *alloc(size_t n)
    {
        void *p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(U)) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        owned.push_back(p); // a null entry marks a failed allocation
        return static_cast<U *>(p);
    }
    void release()
    {
        if (stepGraph) cudaGraphExecDestroy(stepGraph);
        if (adjointGraph) cudaGraphExecDestroy(adjointGraph);
        stepGraph = adjointGraph = nullptr;
        for (void *p : owned)
            if (p) cudaFree(p);
        owned.clear();
    }
};

void copyAsync(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    if (bytes) cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st);
}

// A kernel of the iterations over `threads`, launched ahead of its predecessor's end.
template <class... P, class... A> void launchDependent(void (*k)(P...), size_t threads, cudaStream_t st, A... args)
{
    cn::launchPdl(k, gridOf(threads), unsigned(kDiffThreads), st, args...);
}

// One substep of the state (g.x, g.v).  With `record` every iteration writes its positions and lambdas to
// the next slot of the iteration states instead of in place, for the adjoint: edges of iteration `it` at
// (itX0, itLE)[it], tets at (itX1, itLT)[it].
template <class T> void runSubstep(Engine<T> &g, bool record, cudaStream_t st)
{
    const DScene<T> &s = g.s;
    const size_t lanes = size_t(s.N) * kLanes;
    P4<T> *cur = record ? g.itX0 : g.x;
    k_dPredict<T><<<gridOf(s.N), kDiffThreads, 0, st>>>(s, g.x, cur, g.v, g.xprev, g.dt);
    for (uint32_t it = 0; it < g.iterations; ++it) {
        const bool last = it + 1u == g.iterations, first = it == 0u;
        P4<T> *done = !record ? g.x : last ? g.x : g.itX0 + size_t(it + 1u) * s.N;
        if (s.E) {
            T *in = record ? g.itLE + size_t(it) * s.E : g.lamE;
            T *out = record && !last ? in + s.E : g.lamE;
            P4<T> *to = record && s.T_ ? g.itX1 + size_t(it) * s.N : done;
            launchDependent(k_dEdges<T>, s.E, st, s, cur, in, out, g.corrE, g.dt, first);
            launchDependent(k_dGather<T, false>, lanes, st, s, cur, to, s.edgeRanges, g.corrE);
            cur = to;
        }
        if (s.T_) {
            T *in = record ? g.itLT + size_t(it) * s.T_ : g.lamT;
            T *out = record && !last ? in + s.T_ : g.lamT;
            launchDependent(k_dTets<T>, s.T_, st, s, cur, g.compliance, in, out, g.corrT, g.dt, first);
            launchDependent(k_dGather<T, false>, lanes, st, s, cur, done, s.tetRanges, g.corrT);
            cur = done;
        }
    }
    if (cur != g.x) copyAsync(g.x, cur, sizeof(P4<T>) * s.N, st); // neither edges nor tets
    k_dVelocity<T><<<gridOf(s.N), kDiffThreads, 0, st>>>(s, g.x, g.xprev, g.v, g.dt);
}

// The substep from (g.x, g.v) with its iteration states, then its adjoint: (g.gX, g.gV) from those of its end
// to those of its start, the compliances' added to g.gCompliance.
template <class T> void runAdjoint(Engine<T> &g, cudaStream_t st)
{
    const DScene<T> &s = g.s;
    const size_t lanes = size_t(s.N) * kLanes;
    runSubstep(g, true, st);
    P4<T> *gA = g.gA, *gB = g.gB; // gA: the adjoint entering the last iteration's output
    k_dVelocityBack<T><<<gridOf(s.N), kDiffThreads, 0, st>>>(s, g.gX, g.gV, gA, g.dt);
    if (s.E) cudaMemsetAsync(g.gLE, 0, sizeof(T) * s.E, st);
    if (s.T_) cudaMemsetAsync(g.gLT, 0, sizeof(T) * s.T_, st);
    for (int it = int(g.iterations) - 1; it >= 0; --it) {
        if (s.T_) {
            const P4<T> *x = (s.E ? g.itX1 : g.itX0) + size_t(it) * s.N;
            launchDependent(k_dTetsBack<T>, s.T_, st, s, x, g.compliance, g.itLT + size_t(it) * s.T_, gA, g.gLT, g.recT,
                            g.gCompliance, g.dt);
            launchDependent(k_dGather<T, true>, lanes, st, s, gA, gB, s.tetRanges, g.recT);
            std::swap(gA, gB);
        }
        if (s.E) {
            launchDependent(k_dEdgesBack<T>, s.E, st, s, g.itX0 + size_t(it) * s.N, g.itLE + size_t(it) * s.E, gA, g.gLE,
                            g.recE, g.dt);
            launchDependent(k_dGather<T, true>, lanes, st, s, gA, gB, s.edgeRanges, g.recE);
            std::swap(gA, gB);
        }
    }
    // predict backwards: (gX, gV) of the substep start
    k_dPredictBack<T><<<gridOf(s.N), kDiffThreads, 0, st>>>(s, gA, g.gV, g.gX, g.gV, g.dt);
}

// Runs one of the two through its graph, captured at first use; on a stream that is itself being captured
// (a caller's graph) the launches go there one by one.
template <class T, class F> cn_status replay(Engine<T> &g, cudaGraphExec_t &exec, cudaStream_t own, cudaStream_t st, F &&enqueue)
{
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) {
        cudaGetLastError(); // the legacy stream beside somebody's capture: not this stream's
        capturing = cudaStreamCaptureStatusNone;
    }
    if (capturing != cudaStreamCaptureStatusNone) {
        enqueue(g, st);
        return CN_OK;
    }
    if (!exec) {
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamBeginCapture(own, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            enqueue(g, own);
            e = cudaStreamEndCapture(own, &graph);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            cudaGetLastError();
            exec = nullptr;
            return setError(CN_ERR_CUDA, std::string("cn_diff: graph capture failed: ") + cudaGetErrorString(e));
        }
    }
    const cudaError_t e = cudaGraphLaunch(exec, st);
    if (e != cudaSuccess) return setError(CN_ERR_CUDA, std::string("cn_diff: ") + cudaGetErrorString(e));
    return CN_OK;
}

template <class T> cn_status step(Engine<T> &g, cudaStream_t own, cudaStream_t st)
{
    return replay(g, g.stepGraph, own, st, [](Engine<T> &e, cudaStream_t on) { runSubstep(e, false, on); });
}

template <class T> cn_status forward(Engine<T> &g, const T *compliance, const P4<T> *x0, const P4<T> *v0, P4<T> *xOut,
                                     P4<T> *vOut, cudaStream_t own, cudaStream_t st)
{
    const size_t nb = sizeof(P4<T>) * g.s.N;
    if (g.s.T_) cudaMemcpyAsync(g.compliance, compliance, sizeof(T) * g.s.T_, cudaMemcpyDefault, st);
    copyAsync(g.x, x0, nb, st);
    copyAsync(g.v, v0, nb, st);
    // corrections start at zero (the solver's upload clears them)
    if (g.s.E) cudaMemsetAsync(g.corrE, 0, sizeof(P4<T>) * 2 * g.s.E, st);
    if (g.s.T_) cudaMemsetAsync(g.corrT, 0, sizeof(P4<T>) * 4 * g.s.T_, st);
    for (uint32_t sub = 0; sub < g.substeps; ++sub) {
        if (sub % g.interval == 0) {
            const size_t c = sub / g.interval;
            copyAsync(g.ckX + c * g.s.N, g.x, nb, st);
            copyAsync(g.ckV + c * g.s.N, g.v, nb, st);
        }
        const cn_status r = step(g, own, st);
        if (r != CN_OK) return r;
    }
    if (xOut) copyAsync(xOut, g.x, nb, st);
    if (vOut) copyAsync(vOut, g.v, nb, st);
    g.forwardDone = true;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return setError(CN_ERR_CUDA, std::string("cn_diff_forward: ") + cudaGetErrorString(e));
    return CN_OK;
}

// The stale-record case of the tet solve (a record kept from an earlier iteration) carries no
// derivative here: it only arises for tets whose four particles are all pinned (their records are
// never applied) or whose denominator vanishes.
template <class T> cn_status backward(Engine<T> &g, const P4<T> *gXOut, const P4<T> *gVOut, T *gCompliance,
                                      P4<T> *gX0, P4<T> *gV0, cudaStream_t own, cudaStream_t st)
{
    if (!g.forwardDone) return setError(CN_ERR_NOT_INITIALIZED, "cn_diff_backward: run cn_diff_forward first");
    const DScene<T> &s = g.s;
    const size_t nb = sizeof(P4<T>) * s.N;
    if (gXOut) copyAsync(g.gX, gXOut, nb, st); else cudaMemsetAsync(g.gX, 0, nb, st);
    if (gVOut) copyAsync(g.gV, gVOut, nb, st); else cudaMemsetAsync(g.gV, 0, nb, st);
    if (s.T_) cudaMemsetAsync(g.gCompliance, 0, sizeof(T) * s.T_, st);
    const uint32_t segments = (g.substeps + g.interval - 1) / g.interval;
    for (int seg = int(segments) - 1; seg >= 0; --seg) {
        const uint32_t first = uint32_t(seg) * g.interval;
        const uint32_t count = std::min(g.interval, g.substeps - first);
        // recompute the segment's substep starts from its checkpoint
        copyAsync(g.x, g.ckX + size_t(seg) * s.N, nb, st);
        copyAsync(g.v, g.ckV + size_t(seg) * s.N, nb, st);
        if (s.E) cudaMemsetAsync(g.corrE, 0, sizeof(P4<T>) * 2 * s.E, st);
        if (s.T_) cudaMemsetAsync(g.corrT, 0, sizeof(P4<T>) * 4 * s.T_, st);
        for (uint32_t k = 0; k < count; ++k) {
            copyAsync(g.segX + size_t(k) * s.N, g.x, nb, st);
            copyAsync(g.segV + size_t(k) * s.N, g.v, nb, st);
            if (k + 1 < count) {
                const cn_status r = step(g, own, st);
                if (r != CN_OK) return r;
            }
        }
        for (int k = int(count) - 1; k >= 0; --k) {
            copyAsync(g.x, g.segX + size_t(k) * s.N, nb, st);
            copyAsync(g.v, g.segV + size_t(k) * s.N, nb, st);
            const cn_status r = replay(g, g.adjointGraph, own, st, [](Engine<T> &e, cudaStream_t on) { runAdjoint(e, on); });
            if (r != CN_OK) return r;
        }
    }
    if (s.T_) cudaMemcpyAsync(gCompliance, g.gCompliance, sizeof(T) * s.T_, cudaMemcpyDefault, st);
    if (gX0) copyAsync(gX0, g.gX, nb, st);
    if (gV0) copyAsync(gV0, g.gV, nb, st);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return setError(CN_ERR_CUDA, std::string("cn_diff_backward: ") + cudaGetErrorString(e));
    return CN_OK;
}

template <class T> cn_status build(Engine<T> &g, const cn_world_soa &w, const cn_diff_desc &d)
{
    const uint32_t N = w.particle_count, E = w.edge_count, TT = w.tet_count;
    DScene<T> &s = g.s;
    s.N = N; s.E = E; s.T_ = TT;
    g.iterations = std::max<uint32_t>(d.iterations, 1u);
    g.substeps = std::max<uint32_t>(d.substeps, 1u);
    g.interval = std::max<uint32_t>(d.checkpoint_interval, 1u);
    g.dt = T(d.substep_dt);
    s.relax = T(d.relaxation);
    for (int k = 0; k < 3; ++k) s.g[k] = T(d.gravity[k]);
    std::vector<T> wv(N), damp(N);
    for (uint32_t i = 0; i < N; ++i) {
        wv[i] = T(w.positions_inv_mass[4 * i + 3]);
        const uint32_t m = w.material_indices[i];
        damp[i] = m < w.contact_material_count ? T(w.contact_materials[4 * m + 2]) : T(0);
    }
    std::vector<uint2> pairs(E);
    std::vector<T> rest(E), ecomp(E);
    std::vector<uint32_t> en(E);
    for (uint32_t e = 0; e < E; ++e) {
        pairs[e] = make_uint2(w.edges[e].particle_a, w.edges[e].particle_b);
        rest[e] = T(w.edges[e].rest_length);
        ecomp[e] = T(w.edges[e].compliance);
        en[e] = w.edges[e].enabled;
    }
    std::vector<uint4> tets(TT);
    std::vector<T> trest(TT);
    for (uint32_t t = 0; t < TT; ++t) {
        const cn_soft_tet &q = w.tets[t];
        tets[t] = make_uint4(q.particle_indices[0], q.particle_indices[1], q.particle_indices[2], q.particle_indices[3]);
        trest[t] = T(q.rest_volume);
    }
    const cn::Incidence eI = cn::buildIncidence(N, E, 2, [&](uint32_t c, uint32_t k) {
        return k == 0 ? w.edges[c].particle_a : w.edges[c].particle_b;
    });
    const cn::Incidence tI = cn::buildIncidence(N, TT, 4, [&](uint32_t c, uint32_t k) { return w.tets[c].particle_indices[k]; });
    auto upload = [&](auto *dst, const auto &vec) {
        if (!vec.empty()) cudaMemcpy(dst, vec.data(), vec.size() * sizeof(vec[0]), cudaMemcpyHostToDevice);
    };
    T *dw = g.template alloc<T>(N), *ddamp = g.template alloc<T>(N);
    uint2 *dpairs = g.template alloc<uint2>(E);
    T *drest = g.template alloc<T>(E), *decomp = g.template alloc<T>(E);
    uint32_t *den = g.template alloc<uint32_t>(E);
    uint4 *dtets = g.template alloc<uint4>(TT);
    T *dtrest = g.template alloc<T>(TT);
    uint2 *eR = g.template alloc<uint2>(N), *tR = g.template alloc<uint2>(N);
    uint32_t *eDst = g.template alloc<uint32_t>(eI.dst.size()), *tDst = g.template alloc<uint32_t>(tI.dst.size());
    g.compliance = g.template alloc<T>(TT); g.gCompliance = g.template alloc<T>(TT);
    const size_t ck = g.substeps / g.interval + 1;
    g.x = g.template alloc<P4<T>>(N); g.v = g.template alloc<P4<T>>(N); g.xprev = g.template alloc<P4<T>>(N);
    g.lamE = g.template alloc<T>(E); g.lamT = g.template alloc<T>(TT);
    g.corrE = g.template alloc<P4<T>>(size_t(E) * 2); g.corrT = g.template alloc<P4<T>>(size_t(TT) * 4);
    g.ckX = g.template alloc<P4<T>>(ck * N); g.ckV = g.template alloc<P4<T>>(ck * N);
    g.segX = g.template alloc<P4<T>>(size_t(g.interval) * N); g.segV = g.template alloc<P4<T>>(size_t(g.interval) * N);
    g.itX0 = g.template alloc<P4<T>>(size_t(g.iterations) * N); g.itX1 = g.template alloc<P4<T>>(size_t(g.iterations) * N);
    g.itLE = g.template alloc<T>(size_t(g.iterations) * E); g.itLT = g.template alloc<T>(size_t(g.iterations) * TT);
    g.gX = g.template alloc<P4<T>>(N); g.gV = g.template alloc<P4<T>>(N);
    g.gA = g.template alloc<P4<T>>(N); g.gB = g.template alloc<P4<T>>(N);
    g.gLE = g.template alloc<T>(E); g.gLT = g.template alloc<T>(TT);
    g.recE = g.template alloc<P4<T>>(size_t(E) * 2); g.recT = g.template alloc<P4<T>>(size_t(TT) * 4);
    for (void *p : g.owned)
        if (!p) return setError(CN_ERR_OUT_OF_MEMORY, "cn_diff_set_scene: device allocation failed");
    upload(dw, wv); upload(ddamp, damp); upload(dpairs, pairs); upload(drest, rest); upload(decomp, ecomp);
    upload(den, en); upload(dtets, tets); upload(dtrest, trest);
    upload(eR, eI.ranges); upload(eDst, eI.dst); upload(tR, tI.ranges); upload(tDst, tI.dst);
    // the first iteration starts from zero lambdas: the adjoint reads them in the first slots, which nothing writes
    cudaMemset(g.itLE, 0, sizeof(T) * std::max<uint32_t>(E, 1u));
    cudaMemset(g.itLT, 0, sizeof(T) * std::max<uint32_t>(TT, 1u));
    s.w = dw; s.damp = ddamp; s.edgePair = dpairs; s.edgeRest = drest; s.edgeCompliance = decomp; s.edgeEnabled = den;
    s.tetIdx = dtets; s.tetRest = dtrest; s.edgeRanges = eR; s.tetRanges = tR;
    s.edgeDst = reinterpret_cast<const uint2 *>(eDst); s.tetDst = reinterpret_cast<const uint4 *>(tDst);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return setError(CN_ERR_CUDA, std::string("cn_diff_set_scene: ") + cudaGetErrorString(e));
    return CN_OK;
}

} // namespace

struct cn_diff {
    cn_diff_desc desc{};
    int device = 0;
    cudaStream_t ownStream = nullptr;
    Engine<float> f32;
    Engine<double> f64;
    bool ready = false;
    uint32_t N = 0, T = 0;
};

extern "C" {

CN_API void cn_diff_desc_defaults(cn_diff_desc *d)
{
    if (!d) return;
    std::memset(d, 0, sizeof(*d));
    d->gravity[1] = -9.81f;
    d->substeps = 32;
    d->iterations = 20;
    d->substep_dt = 1.0f / 60.0f / 32.0f;
    d->relaxation = 0.2f;
    d->checkpoint_interval = 8;
    d->precision = 4;
}

CN_API cn_status cn_diff_create(const cn_diff_desc *d, int device, cn_diff **out)
{
    if (!d || !out) return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_create: null argument");
    *out = nullptr;
    if (d->precision != 4 && d->precision != 8) return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_create: precision is 4 or 8");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return setError(CN_ERR_NO_DEVICE, "cn_diff_create: no CUDA device");
    }
    if (device < 0 || device >= count) return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_create: bad device");
    auto *g = new cn_diff();
    g->desc = *d;
    g->device = device;
    cudaSetDevice(device);
    cudaStreamCreateWithFlags(&g->ownStream, cudaStreamNonBlocking);
    *out = g;
    return CN_OK;
}

CN_API void cn_diff_destroy(cn_diff *g)
{
    if (!g) return;
    cudaSetDevice(g->device);
    cudaDeviceSynchronize();
    g->f32.release();
    g->f64.release();
    if (g->ownStream) cudaStreamDestroy(g->ownStream);
    delete g;
}

CN_API cn_status cn_diff_set_scene(cn_diff *g, const cn_world_soa *w)
{
    if (!g || !w) return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_set_scene: null argument");
    if (w->bend_count || w->dihedral_count || w->strand_segment_count || w->strand_joint_count ||
        w->strand_distance_count || w->collider_count)
        return setError(CN_ERR_UNSUPPORTED, "cn_diff_set_scene: the differentiable rollout covers edges and tets "
                                            "without colliders");
    for (uint32_t i = 0; i < w->particle_count; ++i)
        if (w->kinds[i] == CN_PARTICLE_FLUID || (w->owner_types && w->owner_types[i] == CN_OWNER_RIGID_BODY))
            return setError(CN_ERR_UNSUPPORTED, "cn_diff_set_scene: fluid or rigid proxy particles");
    cudaSetDevice(g->device);
    cudaDeviceSynchronize();
    g->f32.release();
    g->f64.release();
    g->f32 = Engine<float>();
    g->f64 = Engine<double>();
    const cn_status st = g->desc.precision == 8 ? build(g->f64, *w, g->desc) : build(g->f32, *w, g->desc);
    if (st != CN_OK) return st;
    g->ready = true;
    g->N = w->particle_count;
    g->T = w->tet_count;
    return CN_OK;
}

CN_API cn_status cn_diff_forward(cn_diff *g, const void *tet_compliance, const void *x0, const void *v0, void *x_out,
                                 void *v_out, void *stream)
{
    if (!g || !g->ready || !tet_compliance || !x0 || !v0)
        return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_forward: no scene or null buffer");
    cudaSetDevice(g->device);
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : g->ownStream;
    if (g->desc.precision == 8)
        return forward(g->f64, static_cast<const double *>(tet_compliance), static_cast<const P4<double> *>(x0),
                       static_cast<const P4<double> *>(v0), static_cast<P4<double> *>(x_out),
                       static_cast<P4<double> *>(v_out), g->ownStream, st);
    return forward(g->f32, static_cast<const float *>(tet_compliance), static_cast<const P4<float> *>(x0),
                   static_cast<const P4<float> *>(v0), static_cast<P4<float> *>(x_out), static_cast<P4<float> *>(v_out),
                   g->ownStream, st);
}

CN_API cn_status cn_diff_backward(cn_diff *g, const void *grad_x_out, const void *grad_v_out, void *grad_tet_compliance,
                                  void *grad_x0, void *grad_v0, void *stream)
{
    if (!g || !g->ready || !grad_tet_compliance)
        return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_backward: no scene or null buffer");
    cudaSetDevice(g->device);
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : g->ownStream;
    if (g->desc.precision == 8)
        return backward(g->f64, static_cast<const P4<double> *>(grad_x_out), static_cast<const P4<double> *>(grad_v_out),
                        static_cast<double *>(grad_tet_compliance), static_cast<P4<double> *>(grad_x0),
                        static_cast<P4<double> *>(grad_v0), g->ownStream, st);
    return backward(g->f32, static_cast<const P4<float> *>(grad_x_out), static_cast<const P4<float> *>(grad_v_out),
                    static_cast<float *>(grad_tet_compliance), static_cast<P4<float> *>(grad_x0),
                    static_cast<P4<float> *>(grad_v0), g->ownStream, st);
}

CN_API cn_status cn_diff_memory(cn_diff *g, uint64_t *bytes)
{
    if (!g || !bytes) return setError(CN_ERR_INVALID_ARGUMENT, "cn_diff_memory: null argument");
    const Engine<float> &a = g->f32;
    const Engine<double> &b = g->f64;
    const size_t es = g->desc.precision == 8 ? 8 : 4;
    const uint32_t iters = g->desc.precision == 8 ? b.iterations : a.iterations;
    const uint32_t subs = g->desc.precision == 8 ? b.substeps : a.substeps;
    const uint32_t interval = g->desc.precision == 8 ? b.interval : a.interval;
    const uint32_t E = g->desc.precision == 8 ? b.s.E : a.s.E;
    const size_t N = g->N, T = g->T;
    // the state saved for the adjoint: checkpoints, one segment, one substep's iterations
    *bytes = uint64_t((subs / interval + 1) * 2 * N * 4 * es + size_t(interval) * 2 * N * 4 * es +
                      size_t(iters) * (2 * N * 4 * es + (E + T) * es));
    return CN_OK;
}

} // extern "C"
