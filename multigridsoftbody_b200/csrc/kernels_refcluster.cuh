// Every iteration of the reference-faithful frame of a body in one launch: of a small one by one thread-block cluster, of
// a larger one by a cooperative launch over every SM.
#pragma once

#include "kernels.cuh"
#include "kernels_mg.cuh"
#include "kernels_twolevel.cuh"

namespace mgsb {
namespace {

// ---------------------------------------------------------------------------
// k_ref_local and k_ref_vertex alternate, 2.8-3.0 us each on a small body whatever
// they do: the latency of a launch, of its loads and of its end.  Here CTA `rank`
// of the cluster owns consecutive vertices and runs all iterations on them:
//   - the tets around its vertices (some of them in other CTAs too), and where
//     each corner's contribution goes, lie in shared memory, one image per CTA,
//     laid out by the host and brought by one bulk copy before the dependency
//     wait; the tets' constants follow it there;
//   - x over the window of vertices that those tets read (contiguous in the
//     numbering) is double buffered: the owner of a vertex stores its new position
//     into the other buffer of every CTA whose window holds it, and one cluster
//     barrier ends the iteration;
//   - contributions are summed in ascending tet order by the vertex's thread, as
//     k_ref_vertex does.
// The functions, their order and so the bits are those of the two kernels, and of
// k_ref_predict, which every CTA applies to its whole window.
// With triangles (the coarse level of the two-level schedule) a CTA also forms the
// pushes of the surface triangles around its vertices (k_ref_tri_dcd).
// ---------------------------------------------------------------------------
// On a body too large for one cluster (kGrid) the same runs as a cooperative launch
// of one CTA per SM: positions go through L2 (two buffers, for the same reason), and
// a barrier over the grid, one atomic add per CTA and one thread of each polling,
// ends the iteration.
constexpr int kRefThreads = 512;   // at most; a thread per own vertex, and tets in turn
constexpr int kRefPolls = 1 << 22;   // of a grid barrier; then the frame is given up and marked non-finite

__device__ __forceinline__ void grid_arrive(int32_t* count) {   // thread 0, behind a barrier of the CTA
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(count) : "memory");
}
__device__ __forceinline__ bool grid_reached(const int32_t* count, int target) {
    for (int polls = 0; polls < kRefPolls; ++polls) {
        int32_t c;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if (c >= target) return true;
    }
    return false;
}

struct RefHead {   // at the start of the image
    int tets, own, first, tris;
    int win_lo, win_n, pad[2];
    int peer_lo[kMaxCluster];   // the CTAs' windows' first vertices
};
struct RefPlan {   // offsets: bytes in the CTA's dynamic shared memory, the same in every CTA
    const unsigned char* image;
    int image_bytes;
    int id;                                  // per tet
    int deg, to;                             // per own vertex: contributions, the CTAs that read it (one bit each)
    int tri, tri_ptr, tri_idx;               // triangles among the window; per own vertex, its triangles
    int corner, slot;                        // per tet, the image's last part (k_ref_image): corners among the window,
                                             // contributions, 0xffff where another CTA owns the vertex
    int inv_a, inv_b, inv_c, win[2], slots, push;   // what the kernel writes: the tets' constants, positions, contributions
    const float4 *from_a, *from_b;           // the constants of all tets
    const float2* from_c;
    int stride;                              // contribution k of own vertex v at slots[k * stride + v]
    int bytes, block, ctas, grid;            // grid: a cooperative launch, not a cluster
    int with_tris;                           // surface triangles that the images hold
    const float* omega;                      // Chebyshev factor of each iteration
    float4* pos[2];                          // grid: the positions that odd and even iterations leave
    int32_t* barrier;                        // grid: arrivals, CTAs that are done; both 0 between launches
};

// The images' corners and contributions, at set-up: contribution k of a vertex is its k-th slot.
__global__ void k_ref_image(RefPlan Q, unsigned char* images, const int4* __restrict__ tets, const int4* __restrict__ slot_of,
                            const int32_t* __restrict__ slot_ptr) {
    unsigned char* image = images + (size_t)blockIdx.x * Q.image_bytes;
    const RefHead& head = *reinterpret_cast<const RefHead*>(image);
    for (int r = threadIdx.x; r < head.tets; r += blockDim.x) {
        const int t = reinterpret_cast<const int32_t*>(image + Q.id)[r];
        const int4 id = __ldg(tets + t), so = __ldg(slot_of + t);
        auto contribution = [&](int i, int at) -> uint16_t {
            const int v = i - head.first;
            if (v < 0 || v >= head.own) return (uint16_t)0xffff;
            return (uint16_t)((at - __ldg(slot_ptr + i / kSlotSlice) - i % kSlotSlice) / kSlotSlice * Q.stride + v);
        };
        reinterpret_cast<ushort4*>(image + Q.corner)[r] =
            make_ushort4((uint16_t)(id.x - head.win_lo), (uint16_t)(id.y - head.win_lo), (uint16_t)(id.z - head.win_lo),
                         (uint16_t)(id.w - head.win_lo));
        reinterpret_cast<ushort4*>(image + Q.slot)[r] = make_ushort4(contribution(id.x, so.x), contribution(id.y, so.y),
                                                                     contribution(id.z, so.z), contribution(id.w, so.w));
    }
}

template <bool kGrid>
__global__ void __launch_bounds__(kRefThreads, 1) k_ref_iterations(
    const RefPlan Q, int iterations, int predict, const RefPredict pa, float4* __restrict__ x, float4* __restrict__ prev,
    float4* __restrict__ s, float4* __restrict__ last, float4* __restrict__ v, const float* __restrict__ fixf, const float* __restrict__ mass,
    const float* __restrict__ vdiag, const SphereSet* __restrict__ sphere_set, float stiffness, int drop_small, float kc,
    float dt, double relax, int with_tris, int last_iter, int32_t* __restrict__ cflag, float* __restrict__ cdepth,
    float* __restrict__ cenergy, int32_t* __restrict__ nonfinite) {
    pdl_trigger();
    extern __shared__ __align__(128) unsigned char smb[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ SphereSet spheres;
    __shared__ int stop;
    const int rank = (int)blockIdx.x, tid = threadIdx.x;   // one cluster, or the grid
    if (tid == 0) {
        stop = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(&bar, (uint32_t)Q.image_bytes);
        bulk_g2s(smb, Q.image + (size_t)rank * Q.image_bytes, (uint32_t)Q.image_bytes, &bar);
    }
    for (int k = tid; k < (int)(sizeof(SphereSet) / 4); k += blockDim.x)
        reinterpret_cast<int32_t*>(&spheres)[k] = reinterpret_cast<const int32_t*>(sphere_set)[k];
    __syncthreads();
    // when the image does not arrive the CTA takes part in the barriers only, and the frame ends marked non-finite
    const bool ok = cta_wait(&bar, 0, kMaxPolls);
    const RefHead& head = *reinterpret_cast<const RefHead*>(smb);
    const int tets = ok ? head.tets : 0, tris = ok && with_tris ? head.tris : 0, own = ok ? head.own : 0;
    // the vertices' threads come last: where the tets leave them free they look for contact meanwhile
    const int vert = tid - ((int)blockDim.x - (own + 31) / 32 * 32);
    const int i = ok ? head.first + vert : 0;
    const bool mine = vert >= 0 && vert < own;
    const float fix = mine ? __ldg(fixf + i) : 0.f, vd = mine ? __ldg(vdiag + i) : 0.f;
    const float dc = mine ? __ldg(mass + i) / (dt * dt) : 0.f;
    const int deg = mine ? reinterpret_cast<const uint16_t*>(smb + Q.deg)[vert] : 0;
    const uint32_t to = mine ? reinterpret_cast<const uint16_t*>(smb + Q.to)[vert] : 0;
    const uint32_t base = smem_u32(smb);
    for (int t = tid; t < tets; t += blockDim.x) {   // written by no kernel of a frame
        const int q = reinterpret_cast<const int32_t*>(smb + Q.id)[t];
        reinterpret_cast<float4*>(smb + Q.inv_a)[t] = __ldg(Q.from_a + q);
        reinterpret_cast<float4*>(smb + Q.inv_b)[t] = __ldg(Q.from_b + q);
        reinterpret_cast<float2*>(smb + Q.inv_c)[t] = __ldg(Q.from_c + q);
    }
    pdl_wait();
    {
        float4* w = reinterpret_cast<float4*>(smb + Q.win[0]);
        const int n = ok ? head.win_n : 0;
        for (int k = tid; k < n; k += blockDim.x) {
            const int g = head.win_lo + k;
            float4 p = x[g];
            if (predict) {
                float4 vel = v[g];
                ref_predict(p, vel, __ldg(fixf + g), pa, dt);
            }
            w[k] = p;
        }
    }
    float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f), pv4 = s4, l4 = s4;   // this thread's vertex: prediction, previous iterate, frame start
    if (mine && predict) {
        l4 = s4 = x[i];
        float4 vel = v[i];
        ref_predict(s4, vel, fix, pa, dt);
        pv4 = s4;
        s[i] = s4;
        last[i] = l4;
    } else if (mine) {
        s4 = s[i];
        pv4 = prev[i];
        l4 = last[i];
    }
    int target = 0;
    // every CTA has read what it needs and written what the others read; false: one did not arrive in time
    auto together = [&]() -> bool {
        if (!kGrid) {
            cluster_arrive();
            cluster_wait();
            return true;
        }
        target += gridDim.x;
        __syncthreads();
        if (tid == 0) {
            grid_arrive(Q.barrier);
            if (!grid_reached(Q.barrier, target)) stop = 1;
        }
        __syncthreads();
        return !stop;
    };
    // cluster: every CTA runs before it is written to; both: x has been read before it is written
    bool on = kGrid && iterations > 1 ? (__syncthreads(), true) : together();
    float4* slots = reinterpret_cast<float4*>(smb + Q.slots);
    for (int it = 0; it < iterations && on; ++it) {
        const float omega = __ldg(Q.omega + it);
        float4* w = reinterpret_cast<float4*>(smb + Q.win[kGrid ? 0 : it & 1]);
        if (kGrid && it > 0) {
            const int n = ok ? head.win_n : 0;
            for (int k = tid; k < n; k += blockDim.x) w[k] = __ldcg(Q.pos[it & 1] + head.win_lo + k);
            __syncthreads();
        }
        RefContact ct;
        const float4 p4 = mine ? w[i - head.win_lo] : s4;
        if (mine && !with_tris) ref_contact(p4, ct, &spheres, kc);
        for (int t = tid; t < tets; t += blockDim.x) {
            const ushort4 id = reinterpret_cast<const ushort4*>(smb + Q.corner)[t];
            const ushort4 so = reinterpret_cast<const ushort4*>(smb + Q.slot)[t];
            float4 out[4];
            ref_tet(reinterpret_cast<const float4*>(smb + Q.inv_a)[t], reinterpret_cast<const float4*>(smb + Q.inv_b)[t],
                    reinterpret_cast<const float2*>(smb + Q.inv_c)[t], w[id.x], w[id.y], w[id.z], w[id.w], stiffness,
                    drop_small, out);
            if (so.x != 0xffff) slots[so.x] = out[0];
            if (so.y != 0xffff) slots[so.y] = out[1];
            if (so.z != 0xffff) slots[so.z] = out[2];
            if (so.w != 0xffff) slots[so.w] = out[3];
        }
        float4* push = reinterpret_cast<float4*>(smb + Q.push);
        for (int f = tid; f < tris; f += blockDim.x) {
            const ushort4 c = reinterpret_cast<const ushort4*>(smb + Q.tri)[f];
            push[f] = ref_tri_push(w[c.x], w[c.y], w[c.z], &spheres);
        }
        __syncthreads();
        if (mine) {
            float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll 4
            for (int k = 0; k < deg; ++k) {
                const float4 c = slots[k * Q.stride + vert];
                fx += c.x; fy += c.y; fz += c.z;
            }
            if (with_tris) {
                float cnt = 0.f, mx = 0.f, my = 0.f, mz = 0.f;
                const uint16_t* ptr = reinterpret_cast<const uint16_t*>(smb + Q.tri_ptr);
                for (int e = ptr[vert]; e < ptr[vert + 1]; ++e) {
                    const float4 q = push[reinterpret_cast<const uint16_t*>(smb + Q.tri_idx)[e]];
                    mx += q.x;
                    my += q.y;
                    mz += q.z;
                    cnt += q.w;
                }
                ct.cd[0] = ct.cd[1] = ct.cd[2] = kc * cnt;
                ct.cf[0] = kc * mx;
                ct.cf[1] = kc * my;
                ct.cf[2] = kc * mz;
                ct.flag = (int)cnt;
            }
            const float4 xn = ref_vertex(p4, s4, pv4, make_float4(fx, fy, fz, 0.f), ct, dc, vd, fix, omega, relax);
            pv4 = p4;
            if (kGrid && it + 1 < iterations) {
                __stcg(Q.pos[(it + 1) & 1] + i, xn);
            } else if (it + 1 < iterations) {
                for (uint32_t m = to; m; m &= m - 1) {
                    const int c = __ffs(m) - 1;
                    cluster_st(cluster_addr(base + Q.win[(it + 1) & 1] + 16 * (i - head.peer_lo[c]), c), xn);
                }
            } else {
                x[i] = xn;
                prev[i] = p4;
                // last_iter: bit 0 = velocity, bit 1 = contact outputs and the finiteness check
                if (last_iter & 1) {
                    v[i] = make_float4((xn.x - l4.x) / dt, (xn.y - l4.y) / dt, (xn.z - l4.z) / dt, 0.f);
                }
                if (last_iter & 2) {
                    cflag[i] = ct.flag;
                    cdepth[i] = ct.depth;
                    cenergy[i] = ct.energy;
                    if (!isfinite(xn.x) || !isfinite(xn.y) || !isfinite(xn.z)) atomicOr(nonfinite, 1);
                }
            }
        }
        if (it + 1 == iterations) break;
        on = together();   // the new positions are there, the contributions have been read
    }
    if (kGrid && tid == 0) {
        if (!on) atomicOr(nonfinite, 1);
        if (atomicAdd(Q.barrier + 1, 1) == (int)gridDim.x - 1) {   // every other CTA has left: ready for the next launch
            Q.barrier[0] = 0;
            Q.barrier[1] = 0;
        }
    }
    if (!ok) {   // a copy that never arrived is waited for again before the CTA ends
        if (tid == 0) atomicOr(nonfinite, 1);
        mbar_wait(&bar, 0, kMaxPolls);
    }
}

}  // namespace
}  // namespace mgsb
