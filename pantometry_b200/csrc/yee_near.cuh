// The near field of an FP32 cavity's soft current, kept in f64.
//
// Why. A soft current drives the field at its edge up and down with every cycle of the pulse, and
// what flows in and out of the edge and its neighbours is many times the net work the source does.
// Stored in f32, those values are rounded on every step while that flow passes through them, and
// the ledger (invariant − work) ends a few 1e-6 of the injected energy away from the f64 run's. A
// numpy emulation of the scheme shows where it comes from: with the six components of a 5³ box of
// lattice nodes around the source kept in f64 (every stencil reading the stored values), the same
// run ends 1e-9 away, against 2e-6 with the whole field in f32.
//
// The rule, in one line: inside the box every value is f64, outside it f32, and every stencil reads
// what is stored. The tiles of yee_tma_step step every node in f32 from the stored values (the box's f32
// roundings included) but leave to block 0 the box's faces, edges and energy terms, the source, and the
// ring: the edges just outside the box whose curl reads a box face. Block 0, which takes no tiles,
//   loads the old f32 field of the box and a node around it, and the box's f64 values,
//   A. forms H⁺ of the box's faces in f64 from the box's f64 H and E (f32 values outside), and of the
//      faces around it in f32 by the tiles' own expression (yee_face_f32), so with their bits,
//   B. forms Eⁿ⁺¹ of the box's edges in f64 from those H⁺, with the source,
//   C. forms the ring in f32 from the H⁺ that is stored (the f32 roundings of the box's faces),
//   D. and gives its sums of the box's energy terms, Joule loss and source work as the tiles' blocks do.
// Nothing of it waits for a tile, so it runs beside them. When the last block did this, after every other
// block had finished, it was a chain of dependent loads at the end of each step: a dielectric 128³ cavity
// ran 51.0 µs a step with a source and 39.3 without one, a vacuum 384³ one 574, a 31 × 27 × 43 one 15.2;
// beside the tiles 37.4, 563 and 13.5 (the loops of the other stages ask no node about the box any more).
// The box and the ring lie inside the walls (one node from them at least), so every component exists at
// every node they hold, every edge is interior and no wall kernel touches it.
//
// The arithmetic of A and B is cavity.rs:1346-1452 with the uniform medium's f64 coefficients (or
// each edge's own f32 gain with MEDIA, the coefficient the update and the energy weight use), the
// soft current as in yee_tma_step.
#pragma once

#include "yee_tma.cuh"

namespace pm {

__device__ __forceinline__ size_t near_lat(const YeeNearArgs& a, int i, int j, int k) {
    return (size_t)i + (size_t)a.L * ((size_t)j + (size_t)a.ny1 * (size_t)k);
}
// Component q's pointer of a lattice set, chosen by a switch: indexing the parameter block's array
// with a runtime index would copy the whole block to local memory.
__device__ __forceinline__ const float* near_comp(const float* const (&lat)[6], int q) {
    switch (q) {
        case 0: return lat[0];
        case 1: return lat[1];
        case 2: return lat[2];
        case 3: return lat[3];
        case 4: return lat[4];
        default: return lat[5];
    }
}
__device__ __forceinline__ float* near_comp(float* const (&lat)[6], int q) {
    switch (q) {
        case 0: return lat[0];
        case 1: return lat[1];
        case 2: return lat[2];
        case 3: return lat[3];
        case 4: return lat[4];
        default: return lat[5];
    }
}
__device__ __forceinline__ const float* near_comp(const float* const (&lat)[3], int q) {
    return q == 0 ? lat[0] : q == 1 ? lat[1] : lat[2];
}
// Seed the box's f64 values from the stored f32 field (after the state was set from outside a step).
static __global__ void yee_near_seed(YeeNearArgs a) {
    const int w = a.w, w3 = w * w * w;
    for (int r = threadIdx.x; r < 6 * w3; r += blockDim.x) {
        const int q = r / w3, l = r - q * w3;
        const int i = a.x0 + l % w, j = a.y0 + (l / w) % w, k = a.z0 + l / (w * w);
        a.nneu[r] = (double)near_comp(a.neu, q)[near_lat(a, i, j, k)];
    }
}

// Block 0's working set, in the tiles' ring of stages: the arguments, the old f32 E of the box and a node
// below and two above it along each axis, H of the box and a node either side, the box's f64 values, H⁺.
struct YeeNearShared {
    static constexpr int W = kNearWidth, W3 = W * W * W, H7 = W + 2, H3 = H7 * H7 * H7, E8 = W + 3, E3 = E8 * E8 * E8;
    YeeNearArgs a;
    double box[6 * W3];
    double hp[3 * H3];  // f64 in the box, an f32 value outside
    float e[3 * E3], h[3 * H3];
};
static_assert(sizeof(YeeNearShared) <= 2 * YeeTmaLayout<3, false>::BYTES, "block 0's working set fits the smallest ring");

// Run by block 0's 256 threads. Local node indices count from x0 − 1, y0 − 1, z0 − 1: the box is 1 .. W.
template <bool SOLID>
__device__ void yee_near_block(YeeNearShared& sh, long long step, double (&acc)[4]) {
    constexpr int W = YeeNearShared::W, W3 = YeeNearShared::W3, H7 = YeeNearShared::H7, H3 = YeeNearShared::H3,
                  E8 = YeeNearShared::E8, E3 = YeeNearShared::E3, T = 256;
    const YeeNearArgs& a = sh.a;
    const int tid = linear_tid();
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const double jsrc = (a.src_i >= 0 && step < a.ncurrent) ? a.current[step] : 0.0;
#pragma unroll
    for (int u = 0; u < (3 * E3 + T - 1) / T; ++u) {
        const int r = tid + T * u, q = r / E3, l = r - q * E3;
        if (r < 3 * E3)
            sh.e[r] = near_comp(a.old, q)[near_lat(a, a.x0 - 1 + l % E8, a.y0 - 1 + (l / E8) % E8, a.z0 - 1 + l / (E8 * E8))];
    }
#pragma unroll
    for (int u = 0; u < (3 * H3 + T - 1) / T; ++u) {
        const int r = tid + T * u, q = r / H3, l = r - q * H3;
        if (r < 3 * H3)
            sh.h[r] = near_comp(a.old, 3 + q)[near_lat(a, a.x0 - 1 + l % H7, a.y0 - 1 + (l / H7) % H7, a.z0 - 1 + l / (H7 * H7))];
    }
#pragma unroll
    for (int u = 0; u < (6 * W3 + T - 1) / T; ++u)
        if (tid + T * u < 6 * W3) sh.box[tid + T * u] = a.nold[tid + T * u];
    __syncthreads();
    auto in = [](int i, int j, int k) {
        return (unsigned)(i - 1) < (unsigned)W && (unsigned)(j - 1) < (unsigned)W && (unsigned)(k - 1) < (unsigned)W;
    };
    auto boxed = [](int q, int i, int j, int k) { return q * W3 + (i - 1) + W * ((j - 1) + W * (k - 1)); };
    auto ef = [&](int q, int i, int j, int k) { return sh.e[q * E3 + i + E8 * (j + E8 * k)]; };  // as stored in f32
    auto ed = [&](int q, int i, int j, int k) {  // as stored: f64 in the box
        return in(i, j, k) ? sh.box[boxed(q, i, j, k)] : (double)ef(q, i, j, k);
    };
    // A. H⁺ of face component q (cavity.rs:1346-1379) with the box's terms of ½μ H⁻·H⁺, and the
    // ½ε|Eⁿ|² terms of its edges (half weights of node-centred boundary samples, cavity.rs:766-772)
    for (int r = tid; r < 3 * H3; r += T) {
        const int q = r / H3, l = r - q * H3, i = l % H7, j = (l / H7) % H7, k = l / (H7 * H7);
        // hx: (ez(j+1) − ez) − (ey(k+1) − ey); hy: (ex(k+1) − ex) − (ez(i+1) − ez);
        // hz: (ey(i+1) − ey) − (ex(j+1) − ex)
        const int c1 = q == 0 ? 2 : q == 1 ? 0 : 1, c2 = q == 0 ? 1 : q == 1 ? 2 : 0;
        const int i1 = q == 2, j1 = q == 0, k1 = q == 1, i2 = q == 1, j2 = q == 2, k2 = q == 0;
        if (!in(i, j, k)) {
            sh.hp[r] = (double)yee_face_f32(sh.h[r], a.chf, ef(c1, i + i1, j + j1, k + k1), ef(c1, i, j, k),
                                            ef(c2, i + i2, j + j2, k + k2), ef(c2, i, j, k));
            continue;
        }
        const int gi = a.x0 - 1 + i, gj = a.y0 - 1 + j, gk = a.z0 - 1 + k;
        const double hi = (gi == 0 || gi == nx) ? 0.5 : 1.0, hj = (gj == 0 || gj == ny) ? 0.5 : 1.0,
                     hk = (gk == 0 || gk == nz) ? 0.5 : 1.0;
        const double was = sh.box[boxed(3 + q, i, j, k)];
        const double curl = (ed(c1, i + i1, j + j1, k + k1) - sh.box[boxed(c1, i, j, k)]) -
                            (ed(c2, i + i2, j + j2, k + k2) - sh.box[boxed(c2, i, j, k)]);
        const double hn = __fma_rn(-a.ch, curl, was);
        sh.hp[r] = hn;
        const size_t n = near_lat(a, gi, gj, gk);
        a.nneu[boxed(3 + q, i, j, k)] = hn;
        near_comp(a.neu, 3 + q)[n] = (float)hn;
        acc[1] += (q == 0 ? hi : q == 1 ? hj : hk) * (hn * was);
        const double e0 = sh.box[boxed(q, i, j, k)];
        const double we = q == 0 ? hj * hk : q == 1 ? hi * hk : hi * hj;
        if (a.media)  // weighted by 1/g, the ε the update uses
            acc[0] += we * (e0 * e0) / (double)near_comp(a.cgain, q)[n];
        else
            acc[0] += we * (e0 * e0);
    }
    __syncthreads();  // H⁺ before any edge reads it
    // B and C: edge component q (cavity.rs:1383-1452) at each node of the box and of its ring, nodes 1 .. W + 1
    constexpr int C6 = W + 1, C3 = C6 * C6 * C6;
    for (int r = tid; r < 3 * C3; r += T) {
        const int q = r / C3, l = r - q * C3, i = 1 + l % C6, j = 1 + (l / C6) % C6, k = 1 + l / (C6 * C6);
        // x reads hz back along y and hy back along z; y reads hx along z and hz along x; z reads hy along x
        // and hx along y
        const int c1 = q == 0 ? 2 : q == 1 ? 0 : 1, c2 = q == 0 ? 1 : q == 1 ? 2 : 0;
        const int i1 = q == 2, j1 = q == 0, k1 = q == 1, i2 = q == 1, j2 = q == 2, k2 = q == 0;
        const bool boxed_node = in(i, j, k);
        if (!boxed_node && !in(i - i1, j - j1, k - k1) && !in(i - i2, j - j2, k - k2)) continue;
        auto hp = [&](int c, int ii, int jj, int kk) { return sh.hp[c * H3 + ii + H7 * (jj + H7 * kk)]; };
        const double p0 = hp(c1, i, j, k), p1 = hp(c1, i - i1, j - j1, k - k1), m0 = hp(c2, i, j, k),
                     m1 = hp(c2, i - i2, j - j2, k - k2);
        const int gi = a.x0 - 1 + i, gj = a.y0 - 1 + j, gk = a.z0 - 1 + k;
        const size_t n = near_lat(a, gi, gj, gk);
        const bool ix = gi >= 1 && gi < nx, iy = gj >= 1 && gj < ny, iz = gk >= 1 && gk < nz;
        const bool interior = q == 0 ? (iy && iz) : q == 1 ? (ix && iz) : (ix && iy);
        const bool hit = SOLID && ((solid_edges(a.solid, nx, ny, gi, gj, gk) >> q) & 1);
        if (boxed_node) {
            const double curl = (p0 - p1) - (m0 - m1);
            const double e0 = sh.box[boxed(q, i, j, k)];
            const double g = a.media ? (double)near_comp(a.cgain, q)[n] : a.gain;
            double v = __fma_rn(g, curl, a.decay * e0);
            if (q == 2 && gi == a.src_i && gj == a.src_j && gk == a.src_k) {
                // soft current: ε dE/dt = ∇×H − J, with the σ term's semi-implicit divisor
                const double e = a.eps_src, ss = a.sig_src;
                // (the product rounded by itself: near its zeros ez is all cancellation, and one rounding
                // here moved its last bits, which thousands of f32 steps then carry through the box)
                v = v - __dmul_rn((a.dt / e) / (1.0 + (ss * a.dt / (2.0 * e))), jsrc);
                acc[3] += -(a.dt * a.volume) * jsrc * (0.5 * (e0 + v));
            }
            v = interior ? v : 0.0;
            if (a.lossy && interior) {
                const double m = 0.5 * (e0 + v);
                acc[2] += a.sig0 * m * m * a.dt * a.volume;
            }
            if (hit) v = 0.0;
            a.nneu[boxed(q, i, j, k)] = v;
            near_comp(a.neu, q)[n] = (float)v;
        } else {
            const float curl = ((float)p0 - (float)p1) - ((float)m0 - (float)m1);
            const float e0 = ef(q, i, j, k), gq = a.media ? near_comp(a.cgain, q)[n] : a.gainf;
            float v = __fmaf_rn(gq, curl, a.decf * e0);
            v = interior ? v : 0.0f;
            if (a.lossy && interior) {
                const double m = 0.5 * ((double)e0 + (double)v);
                acc[2] += a.sig0 * m * m * a.dt * a.volume;
            }
            near_comp(a.neu, q)[n] = hit ? 0.0f : v;
        }
    }
}

}  // namespace pm
