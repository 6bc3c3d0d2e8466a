// solve_wide.cuh — the sweeps with each particle shared by L adjacent lanes,
// for particle counts too small to fill the GPU with one thread each.
// Included by solve.cu, whose device functions it uses.
//
// With one thread per particle a sweep's time has a floor: one particle's
// walk, ~45 neighbours one after another, each a round trip to L2 and a
// chain of square roots and divisions (37 us for the forces of 1,620
// particles and 51 us for 16,384, on a GPU that does a million in 490 us).
// Here the L lanes of a particle form L pairs' terms at once and add them in
// list order (wide.cuh), so every result is the one-thread sweep's, bit for
// bit.

// Walks the list of the group's particle, L entries at a time: each lane
// loads one entry and its neighbour's record and calls terms(scale, record)
// to fill t[R]; fold() follows with the terms of all lanes in `rows`. The
// next chunk's entries are asked for before this chunk's records are used.
template <int L, int R, class T, class Load, class Terms, class Fold>
__device__ __forceinline__ void walk_wide(const uint2 *__restrict__ nbr, uint32_t n, const WideLane &w, uint32_t cnt,
                                          float (*rows)[kRowOf<float>], Load load, Terms terms, Fold fold) {
    const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
    const uint32_t at = threadIdx.x & 31u;
    uint2 e = w.lane < cnt ? list_ld(&nbr[(size_t)w.lane * n + w.i]) : make_uint2(w.i, 0u);
    for (uint32_t k = 0; k < most; k += L) {
        const T rec = load(e.x);
        const bool ok = k + w.lane < cnt;
        const float scale = __uint_as_float(e.y);
        const uint32_t next = k + L + w.lane;
        e = next < cnt ? list_ld(&nbr[(size_t)next * n + w.i]) : make_uint2(w.i, 0u);
        float t[R];
        if (ok) {
            terms(scale, rec, t);
        } else {
#pragma unroll
            for (int a = 0; a < R; ++a) t[a] = 0.0f;
        }
#pragma unroll
        for (int a = 0; a < R; ++a) rows[a][at] = t[a];
        __syncwarp();
        fold();
        __syncwarp();
    }
}

// ---- density_div ------------------------------------------------------------
// The lanes form the nine stencil rows' ranges, then take the rows'
// candidates L at a time in stencil order; a ballot gives each hit its place
// in the particle's staged list. The staged hits are then processed L at a
// time, and the boundary's polynomials are spread over the lanes.
__device__ __forceinline__ float axis_of(F3 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

template <bool kB, int L>
__global__ void __launch_bounds__(kWideThreads) k_density_wide(const __grid_constant__ Geo g, SimBufs b, int slot) {
    constexpr int G = 32 / L, U = kWideLoads<L>;
    __shared__ __align__(16) float s_rows[kWideWarps][7][kRowOf<float>];
    __shared__ uint32_t s_hit[kWideWarps][G][kWideCap<L>];
    __shared__ uint32_t s_beg[kWideWarps][G][9], s_len[kWideWarps][G][9];
    const uint32_t n = g.n, warp = threadIdx.x >> 5, at = threadIdx.x & 31u;
    const WideLane w = wide_lane<L>(n);
    const uint32_t i = w.i, bi = box_index<kB>(g, i);
    const DevParams &P = params_ref<kB>(g, bi);
    const KernelConsts K = kernel_consts(P);
    const F3 pos = xyz(__ldg(&b.wpos[i]));
    const F3 vel = xyz(__ldg(&b.wvel[i]));
    const uint32_t cap = P.nbr_cap;
    uint32_t *beg = s_beg[warp][w.group], *len = s_len[warp][w.group], *hit = s_hit[warp][w.group];
    {
        const Stencil t = stencil_of(P, pos);
        const uint32_t base = cell_base_of<kB>(g, bi);
        for (uint32_t r = w.lane; r < 9u; r += L) {
            uint32_t s = 0, e = 0;
            const bool any = w.live && stencil_row<(int)kSimSlabs>(P, base, b.starts, n, t, (int)(r / 3u) - 1,
                                                                   (int)(r % 3u) - 1, s, e);
            beg[r] = s;
            len[r] = any ? e - s : 0u;
        }
    }
    __syncwarp();
    WideRows c(beg, len, w.lane);
    const uint32_t mine = group_mask<L>(w);
    const uint32_t before = mine & ((1u << at) - 1u);
    WideSums<float, L, 7> sums;
    if (w.lane == 0) sums.acc[0] = P.sigma;  // the self term W(0), sim_solve.wgsl:426
    uint32_t found = 0;
    bool more = true;
    while (__any_sync(0xffffffffu, more)) {
        uint32_t staged = 0;
        while (__any_sync(0xffffffffu, more && staged < kWideStage)) {
            const bool scan = more && staged < kWideStage;
            uint32_t j[U];
            float4 pc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                j[u] = scan && c.any() ? c.at() : i;  // i: nothing (a particle is not its own neighbour)
                pc[u] = __ldg(&b.wpos[j[u]]);
                if (scan) c.next<L>();
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const F3 x = pos - xyz(pc[u]);
                const bool is = j[u] != i && dot(x, x) < K.support_sq;
                const uint32_t hits = __ballot_sync(0xffffffffu, is);
                if (is) hit[staged + __popc(hits & before)] = j[u];
                staged += __popc(hits & mine);
            }
            // the group's first lane has the group's earliest candidate
            const uint32_t row0 = __shfl_sync(0xffffffffu, c.row, 0, L);
            if (scan) more = row0 < 9u;
        }
        __syncwarp();
        const uint32_t most = __reduce_max_sync(0xffffffffu, staged);
        for (uint32_t h0 = 0; h0 < most; h0 += L) {
            const uint32_t h = h0 + w.lane;
            float t[7];
#pragma unroll
            for (int a = 0; a < 7; ++a) t[a] = 0.0f;
            if (h < staged) {
                const uint32_t jj = hit[h];
                const F3 x = pos - xyz(__ldg(&b.wpos[jj]));
                const float4 vj = __ldg(&b.wvel[jj]);
                const float r = sqrtf(dot(x, x));
                const float q = r * K.inv_h;
                t[0] = kernel_q(K, q);
                const float wn = fmaxf(1.0f - q, 0.0f);
                t[1] = wn * wn * wn;
                const float gs = grad_scale(K, r, q);
                const F3 gw = gs * x;
                t[2] = gw.x;
                t[3] = gw.y;
                t[4] = gw.z;
                t[5] = dot(gw, gw);
                t[6] = dot(vel - xyz(vj), gw);
                const uint32_t idx = found + h;
                if (idx < cap) b.nbr[(size_t)idx * n + i] = make_uint2(jj, __float_as_uint(gs));
            }
#pragma unroll
            for (int a = 0; a < 7; ++a) s_rows[warp][a][at] = t[a];
            __syncwarp();
            sums.add(s_rows[warp], w);
            __syncwarp();
        }
        found += staged;
    }
    DensitySums d;
    d.w_sum = sums.template get<0>();
    d.rho_near = sums.template get<1>();
    d.grad_sum = f3(sums.template get<2>(), sums.template get<3>(), sums.template get<4>());
    d.grad_sq = sums.template get<5>();
    d.drho = sums.template get<6>();

    // the boundary: wall q (axis q % 3, low or high side q / 3) and edge q
    // (axes xy, xz, yz by q / 4; sides by its low two bits), then summed in
    // wall_density / wedge_sum / wall_grad_sum's order
    const F3 tl = (pos - wall_lo(P)) * P.inv_h;
    const F3 th = (wall_hi(P) - pos) * P.inv_h;
    constexpr int kWallPer = (6 + L - 1) / L, kEdgePer = (12 + L - 1) / L;
    float wd[kWallPer], wgr[kWallPer], edge[kEdgePer];
#pragma unroll
    for (int p = 0; p < kWallPer; ++p) {
        const int q = (int)w.lane + p * L;
        wd[p] = wgr[p] = 0.0f;
        if (q < 6) {
            const int a = q % 3, c1 = a == 0 ? 1 : 0, c2 = a == 2 ? 1 : 2;
            const float t = axis_of(q < 3 ? tl : th, a);
            wd[p] = wall_density(t);
            wgr[p] = wall_gradient(t) + wedge_dsum(t, axis_of(tl, c1), axis_of(th, c1), axis_of(tl, c2), axis_of(th, c2));
        }
    }
#pragma unroll
    for (int p = 0; p < kEdgePer; ++p) {
        const int q = (int)w.lane + p * L;
        edge[p] = 0.0f;
        if (q < 12) {
            const int a = q / 4 == 2 ? 1 : 0, c = q / 4 == 0 ? 1 : 2;
            edge[p] = wedge(axis_of((q & 2) ? th : tl, a), axis_of((q & 1) ? th : tl, c));
        }
    }
    float D[6], S[6], E[12];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        D[q] = __shfl_sync(0xffffffffu, wd[q / L], q % L, L);
        S[q] = __shfl_sync(0xffffffffu, wgr[q / L], q % L, L);
    }
#pragma unroll
    for (int q = 0; q < 12; ++q) E[q] = __shfl_sync(0xffffffffu, edge[q / L], q % L, L);
    unsigned long long term = 0;
    if (w.live && w.lane == 0) {
        float fill = 0.0f;
        fill += D[0] + D[3];
        fill += D[1] + D[4];
        fill += D[2] + D[5];
        float ws = E[0] + E[1] + E[2] + E[3];
        ws += E[4] + E[5] + E[6] + E[7];
        ws += E[8] + E[9] + E[10] + E[11];
        fill -= ws;
        const float scale = P.rho0 * P.inv_h;
        F3 wg = f3(0.f, 0.f, 0.f);
        wg.x -= scale * S[0];
        wg.x += scale * S[3];
        wg.y -= scale * S[1];
        wg.y += scale * S[4];
        wg.z -= scale * S[2];
        wg.z += scale * S[5];
        b.nbr_n[i] = found < cap ? found : cap;
        if (found > cap) atomicAdd(&g.solve[bi].nbr_over, found - cap);
        term = density_finish(g, b, P, bi, i, pos, vel, d, fill, wg);
    }
    add_term<kB>(&g.solve[bi].acc_div[slot], term);
}

// ---- the list sweeps ----------------------------------------------------------
// divergence_sum over the group's lanes.
template <int L>
__device__ __forceinline__ float divergence_wide(const SimBufs &b, uint32_t n, const WideLane &w, bool on,
                                                 float (*rows)[kRowOf<float>]) {
    const F3 pos = xyz(__ldg(&b.wpos[w.i]));
    const F3 vel = xyz(__ldg(&b.wvel[w.i]));
    WideSums<float, L, 1> sums;
    walk_wide<L, 1, PosVel>(
        b.nbr, n, w, on ? __ldg(&b.nbr_n[w.i]) : 0u, rows,
        [&](uint32_t j) { return PosVel{__ldg(&b.wpos[j]), __ldg(&b.wvel[j])}; },
        [&](float gs, const PosVel &q, float *t) { t[0] = dot(vel - xyz(q.v), pair_grad(gs, pos, q.p)); },
        [&] { sums.add(rows, w); });
    return sums.template get<0>();
}

template <bool kB, int L>
__global__ void __launch_bounds__(kWideThreads) k_div_kappa_wide(Geo g, SimBufs b, int slot, int gate) {
    __shared__ __align__(16) float s_rows[kWideWarps][1][kRowOf<float>];
    const WideLane w = wide_lane<L>(g.n);
    const uint32_t bi = box_index<kB>(g, w.i);
    const bool on = w.live && !gated_out<kB>(g, bi, gate);
    const float drho = divergence_wide<L>(b, g.n, w, on, s_rows[threadIdx.x >> 5]);
    unsigned long long term = 0;
    if (on && w.lane == 0)
        term = div_kappa_finish(g, b, params_ref<kB>(g, bi), bi, w.i, g.st[bi].s.dt, xyz(__ldg(&b.wpos[w.i])), xyz(__ldg(&b.wvel[w.i])), drho);
    add_term<kB>(&g.solve[bi].acc_div[slot], term);
}

template <bool kB, int L>
__global__ void __launch_bounds__(kWideThreads) k_den_kappa_wide(Geo g, SimBufs b, int slot, int gate) {
    __shared__ __align__(16) float s_rows[kWideWarps][1][kRowOf<float>];
    const WideLane w = wide_lane<L>(g.n);
    const uint32_t bi = box_index<kB>(g, w.i);
    const bool on = w.live && !gated_out<kB>(g, bi, gate);
    const float drho = divergence_wide<L>(b, g.n, w, on, s_rows[threadIdx.x >> 5]);
    unsigned long long term = 0;
    if (on && w.lane == 0)
        term = den_kappa_finish(g, b, params_ref<kB>(g, bi), bi, w.i, g.st[bi].s.dt, xyz(__ldg(&b.wpos[w.i])), xyz(__ldg(&b.wvel[w.i])), drho);
    add_term<kB>(&g.solve[bi].acc_den[slot], term);
}

template <bool kB, int L>
__global__ void __launch_bounds__(kWideThreads) k_apply_wide(Geo g, SimBufs b, int add_pressure, int gate) {
    __shared__ __align__(16) float s_rows[kWideWarps][3][kRowOf<float>];
    const WideLane w = wide_lane<L>(g.n);
    const uint32_t bi = box_index<kB>(g, w.i);
    const bool on = w.live && !gated_out<kB>(g, bi, gate);
    const F3 pos = xyz(__ldg(&b.wpos[w.i]));
    const float kd_i = b.kd[w.i];
    float(*rows)[kRowOf<float>] = s_rows[threadIdx.x >> 5];
    WideSums<float, L, 3> sums;
    walk_wide<L, 3, float4>(
        b.nbr, g.n, w, on ? __ldg(&b.nbr_n[w.i]) : 0u, rows, [&](uint32_t j) { return __ldg(&b.wpk[j]); },
        [&](float gs, const float4 &q, float *t) {
            const F3 v = (kd_i + q.w) * pair_grad(gs, pos, q);
            t[0] = v.x;
            t[1] = v.y;
            t[2] = v.z;
        },
        [&] { sums.add(rows, w); });
    const F3 total = f3(sums.template get<0>(), sums.template get<1>(), sums.template get<2>());
    if (on && w.lane == 0) apply_finish(g, b, params_ref<kB>(g, bi).mass, bi, w.i, kd_i, total, add_pressure);
}

// Rows of the forces: visc, blend, near, tension, push (three each), the
// divergence, then the heat's two parts, which one lane adds in turn.
template <bool kB, bool kDiv, int L>
__global__ void __launch_bounds__(kWideThreads) k_forces_wide(Geo g, SimBufs b, int slot, int gate) {
    __shared__ __align__(16) float s_rows[kWideWarps][18][kRowOf<float>];
    const WideLane w = wide_lane<L>(g.n);
    const uint32_t bi = box_index<kB>(g, w.i);
    const bool on = w.live && !(kDiv && gated_out<kB>(g, bi, gate));
    const DevParams &P = params_ref<kB>(g, bi);
    const ForceCtx c = force_ctx(b, P, w.i);
    float(*rows)[kRowOf<float>] = s_rows[threadIdx.x >> 5];
    WideSums<float, L, 16> sums;
    float heat = 0.0f;
    walk_wide<L, 18, Nbr3>(
        b.nbr, g.n, w, on ? __ldg(&b.nbr_n[w.i]) : 0u, rows,
        [&](uint32_t j) { return Nbr3{__ldg(&b.posm[j]), __ldg(&b.wvel[j]), __ldg(&b.aux[j])}; },
        [&](float gs, const Nbr3 &q, float *t) {
            const ForceTerms f = force_pair<kDiv>(c, gs, q);
            const F3 v[5] = {f.visc, -f.blend, f.near, -f.tension, f.push};
#pragma unroll
            for (int a = 0; a < 5; ++a) {
                t[3 * a] = v[a].x;
                t[3 * a + 1] = v[a].y;
                t[3 * a + 2] = v[a].z;
            }
            t[15] = f.drho;
            t[16] = f.heat_in;
            t[17] = -f.heat_out;
        },
        [&] {
            sums.add(rows, w);
            if (w.lane == 0) {
#pragma unroll
                for (int e = 0; e < L; e += 4) {
                    const float4 in = *reinterpret_cast<const float4 *>(rows[16] + w.group * L + e);
                    const float4 out = *reinterpret_cast<const float4 *>(rows[17] + w.group * L + e);
                    heat += in.x;
                    heat += out.x;
                    heat += in.y;
                    heat += out.y;
                    heat += in.z;
                    heat += out.z;
                    heat += in.w;
                    heat += out.w;
                }
            }
        });
    ForceSums s;
    s.visc = f3(sums.template get<0>(), sums.template get<1>(), sums.template get<2>());
    s.blend = f3(sums.template get<3>(), sums.template get<4>(), sums.template get<5>());
    s.near = f3(sums.template get<6>(), sums.template get<7>(), sums.template get<8>());
    s.tension = f3(sums.template get<9>(), sums.template get<10>(), sums.template get<11>());
    s.push = f3(sums.template get<12>(), sums.template get<13>(), sums.template get<14>());
    s.drho = sums.template get<15>();
    s.heat = heat;
    unsigned long long term = 0;
    if (on && w.lane == 0) term = force_finish<kDiv>(g, b, P, bi, w.i, c, s);
    if (kDiv) add_term<kB>(&g.solve[bi].acc_div[slot], term);
}
