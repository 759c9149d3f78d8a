// engine_adjoint.cu — parameter updates and the forward / backward passes of the adjoint
// (kernels in k_adjoint.cu).  No counterpart in the reference.
//
// Forward: a fresh render of R rounds (state cleared) through the ordinary round, recording per
// round the seed, and per pixel the search radius² and the SPPM ratio its gather applied; returns
// the linear image radiance/R + flux/(π r² N).  Backward: for each round, restores its seed,
// re-creates its hit points and photons with the ordinary kernels (the emit pass also keeps the
// unquantised photon power), then runs the gather adjoint and the camera- and photon-path replays.
// Nothing per path vertex is stored between the passes.  Any later round, gather, state write or
// parameter change invalidates the recording.  The round whose buffers are still as its passes left them
// (adj_live: after a forward pass its last round) is not rendered again: a one-round step saves a camera,
// shadow, photon and sort pass: 1.9 ms when it was made, for the 512 x 512 atrium at 2^20 photons.
#include "engine.hpp"

#include <cstring>

namespace phx {

#define CK(x)                                                                                                          \
    do {                                                                                                               \
        cudaError_t e_ = (x);                                                                                          \
        if (e_ != cudaSuccess)                                                                                         \
            return fail(PHX_E_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));                                  \
    } while (0)

uint32_t Engine::n_params() const {
    return sc.size() == 1 ? 4 * (uint32_t)sc[0].mats.size() + 3 * (uint32_t)sc[0].lights.size() : 0;
}

int Engine::set_materials(const phx_material *m, uint32_t n) {
    if (sc.size() != 1)
        return fail(PHX_E_UNSUPPORTED, "materials can only be replaced on single-scene contexts");
    SceneSlot &S = sc[0];
    if (!m || n != S.mats.size())
        return fail(PHX_E_INVALID, "material count differs from the scene's");
    for (uint32_t i = 0; i < n; i++) {
        const phx_material &a = S.mats[i], &b = m[i];
        if (a.diff_index != b.diff_index || a.emis_index != b.emis_index || a.norm_index != b.norm_index ||
            a.occlusion_index != b.occlusion_index || a.metal_rough_index != b.metal_rough_index ||
            a.transmission_index != b.transmission_index)
            return fail(PHX_E_INVALID, "texture indices of a material cannot change");
    }
    adjoint_invalidate();
    CK(cudaStreamSynchronize(st));
    CK(cudaMemcpy(S.bufs[9].p, m, sizeof(phx_material) * n, cudaMemcpyHostToDevice));
    S.mats.assign(m, m + n);
    S.desc.any_transmissive = 0;
    for (const auto &mm : S.mats)
        if (!(mm.transmission < 1e-5f)) // not blocking a shadow ray (NaN included)
            S.desc.any_transmissive = 1;
    invalidate_graph(); // the shadow kernel captured for the scene's kind may no longer fit
    return upload_descs();
}

int Engine::set_lights(const phx_light *l, uint32_t n) {
    if (sc.size() != 1)
        return fail(PHX_E_UNSUPPORTED, "lights can only be replaced on single-scene contexts");
    SceneSlot &S = sc[0];
    if ((n && !l) || n != S.lights.size())
        return fail(PHX_E_INVALID, "light count differs from the scene's");
    for (uint32_t i = 0; i < n; i++)
        if (l[i].kind != S.lights[i].kind ||
            (l[i].kind == PHX_LIGHT_TEXTURED && std::memcmp(&l[i].aux, &S.lights[i].aux, sizeof(phx_f4)) != 0))
            return fail(PHX_E_INVALID, "light kinds and emissive-triangle ranges cannot change");
    if (n == 0)
        return PHX_OK;
    adjoint_invalidate();
    std::vector<float> lum(n);
    lum_pref_sum(l, n, lum.data()); // scene_data.cpp:14-23
    CK(cudaStreamSynchronize(st));
    CK(cudaMemcpy(S.bufs[13].p, l, sizeof(phx_light) * n, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(S.bufs[14].p, lum.data(), 4 * (size_t)n, cudaMemcpyHostToDevice));
    S.lights.assign(l, l + n);
    // the tree's boxes are made for rays starting within box_reach: a light moved farther away than any
    // at set-up gets the reference's margin back (lights that only change power never do)
    if (S.box_reach > 0.0f && !(ray_reach(S.geom_reach, l, n) <= S.box_reach)) {
        CK(bvh_device_loosen(S.bufs[0].as<float>(), S.trav_inner, S.desc.wide != 0, st));
        CK(cudaStreamSynchronize(st));
        S.box_reach = 0.0f;
    }
    S.desc.total_lum = lum[n - 1]; // shading.cpp:26
    S.desc.light_draws = light_sample_draws(l, n, S.desc.total_lum);
    invalidate_graph(); // the captured shadow stage depends on the draw count
    return upload_descs();
}

int Engine::adjoint_forward(uint32_t rounds, float *image) {
    if (sc.size() != 1 || shard.world > 1)
        return fail(PHX_E_UNSUPPORTED, "the adjoint is only available on single-scene, unsharded contexts");
    if (rounds == 0 || rounds > 4096)
        return fail(PHX_E_INVALID, "rounds must be 1..4096");
    SceneSlot &S = sc[0];
    const uint32_t P = total_pixels;
    const size_t rp = (size_t)rounds * P;
    int r;
    if ((r = ensure(adj_seeds, 4 * (size_t)rounds)) || (r = ensure(adj_r2, 4 * rp)) ||
        (r = ensure(adj_ratio, 4 * rp)) || (r = ensure(adj_k, 4 * rp)) || (r = ensure(adj_img, 12 * (size_t)P)))
        return r;
    // The photons' unquantised power (16 bytes a photon slot), which only the backward pass reads.  Where it
    // does not fit, the forward pass goes without it and the backward pass renders the last round again.
    const bool with_power = (adj_slot_pow.p && adj_slot_pow.bytes >= 16 * total_slots) ||
                            adj_slot_pow.alloc(16 * total_slots) == PHX_OK;
    adj_ready = false;
    adj_live = ADJ_NO_ROUND;
    CK(cudaStreamSynchronize(st));
    CK(cudaMemsetAsync(flux.p, 0, 16 * (size_t)P, st));
    CK(cudaMemsetAsync(weight.p, 0, 4 * (size_t)P, st));
    CK(cudaMemsetAsync(radiance.p, 0, 16 * (size_t)P, st));
    S.rounds = 0;
    S.total_emitted = 0;
    in_adjoint = true;
    for (uint32_t n = 0; n < rounds; n++) {
        rec_r2 = adj_r2.as<float>() + (size_t)n * P;
        rec_ratio = adj_ratio.as<float>() + (size_t)n * P;
        r = plain_round();
        if (!r && cudaMemcpyAsync(adj_seeds.as<u32>() + n, d_seeds.p, 4, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            r = fail(PHX_E_CUDA, "seed copy failed");
        if (r) {
            rec_r2 = rec_ratio = nullptr;
            in_adjoint = false;
            return r;
        }
    }
    rec_r2 = rec_ratio = nullptr;
    in_adjoint = false;
    const float inv_n = 1.0f / ((float)S.prm.photons_per_round * (float)rounds);
    launch_adj_image(flux.as<float4>(), radiance.as<float4>(), P, 1.0f / (float)rounds, inv_n, adj_img.as<float>(), st);
    CK(cudaGetLastError());
    if (image)
        CK(cudaMemcpyAsync(image, adj_img.p, 12 * (size_t)P, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    adj_rounds = rounds;
    adj_ready = true;
    adj_k_ready = false;
    if (with_power)
        adj_live = rounds - 1; // its hit points, samples and photons are in the buffers
    return PHX_OK;
}

int Engine::adjoint_backward(const float *dl_dimage, float *grad, uint32_t n_grad) {
    if (sc.size() != 1)
        return fail(PHX_E_UNSUPPORTED, "the adjoint is only available on single-scene contexts");
    if (!adj_ready)
        return fail(PHX_E_STATE, "adjoint_backward needs an adjoint_forward with no round, gather, state write or "
                                 "parameter change in between");
    const uint32_t np = n_params();
    if (!dl_dimage || !grad || n_grad < np)
        return fail(PHX_E_INVALID, "need dL/dI for every pixel and room for every parameter");
    SceneSlot &S = sc[0];
    const uint32_t P = total_pixels, R = adj_rounds;
    int r;
    if ((r = ensure(adj_g, 16 * (size_t)P)) || (r = ensure(adj_gT, 16 * (size_t)P)) ||
        (r = ensure(adj_gA, 16 * (size_t)P)) || (r = ensure(adj_gphi, 16 * max_photons)) ||
        (r = ensure(adj_slot_pow, 16 * total_slots)) || (r = ensure(adj_ph_pow, 16 * max_photons)) ||
        (r = ensure(adj_grad, 8 * (size_t)std::max(np, 1u))) || (r = ensure(adj_paths, 4 * ((size_t)total_emit + 1))))
        return r;
    CK(cudaStreamSynchronize(st));
    // the image buffer is free after the forward pass
    CK(cudaMemcpyAsync(adj_img.p, dl_dimage, 12 * (size_t)P, cudaMemcpyHostToDevice, st));
    launch_adj_begin(adj_img.as<float>(), adj_g.as<float4>(), P, st);
    if (!adj_k_ready) {
        const float inv_n = 1.0f / ((float)S.prm.photons_per_round * (float)R);
        launch_adj_scale(adj_ratio.as<float>(), adj_k.as<float>(), flux.as<float4>(), P, R, inv_n, st);
        adj_k_ready = true;
    }
    CK(cudaMemsetAsync(adj_grad.p, 0, 8 * (size_t)std::max(np, 1u), st));
    AdjBufs ab{};
    ab.g_img = adj_g.as<float4>();
    ab.gT = adj_gT.as<float4>();
    ab.gA = adj_gA.as<float4>();
    ab.gphi = adj_gphi.as<float4>();
    ab.ph_pow = adj_ph_pow.as<float4>();
    ab.offsets = offsets.as<u32>();
    ab.grad = adj_grad.as<double>();
    ab.paths = adj_paths.as<u32>();
    ab.n_paths = adj_paths.as<u32>() + total_emit;
    ab.n_params = np;
    ab.n_mat = (u32)S.mats.size();
    ab.inv_rounds = 1.0f / (float)R;
    ab.block_sums = 4 * (size_t)np <= 32768 ? 1u : 0u;
    ab.tr = trace_out(rs0);
    ab.same_samples = one_sample() && S.desc.light_draws == 1 ? S.desc.direct_samples : 0u;
    ab.occluders = S.desc.any_transmissive;
    in_adjoint = true;
    // The round still in the buffers (the forward pass's last one, unless a pass was run since) goes
    // first and is not rendered again; the others follow.
    const uint32_t live = adj_live;
    for (uint32_t k = 0; k < R && !r; k++) {
        const uint32_t n = live >= R ? k : k == 0 ? live : k <= live ? k - 1 : k;
        if (cudaMemcpyAsync(d_seeds.p, adj_seeds.as<u32>() + n, 4, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
            r = fail(PHX_E_CUDA, "seed copy failed");
            break;
        }
        if (n != live) {
            enq_trace_side();
            enq_emit();
            enq_hash_sort();
            join_side();
        }
        adj_live = n;
        // the photons' unquantised power, in canonical order like the photons
        launch_compact_pow(lc(), adj_slot_pow.as<float4>(), counts.as<u32>(), offsets.as<u32>(),
                           adj_ph_pow.as<float4>(), st);
        launch_adj_clear(adj_gphi.as<float4>(), d_ntotal.as<u32>(), max_photons, st);
        ab.kscale = adj_k.as<float>() + (size_t)n * P;
        ab.r2 = adj_r2.as<float>() + (size_t)n * P;
        ab.perm = perm;
        GatherBufs gbuf{hp[0].as<float4>(), hp[1].as<float4>(), hp[2].as<float4>(), hp[3].as<float4>(),
                        hp[4].as<float4>(), hp[5].as<float4>(), s_posdir.as<float4>(), s_power.as<u32>(),
                        s_dir.as<float4>(), s_pow.as<float4>(), cell_start.as<u32>(), (u32)max_photons,
                        flux.as<float4>(), weight.as<float>(), radiance.as<float4>(), nullptr, nullptr,
                        rs0.order};
        launch_gather_adj(lc(), gbuf, ab, st);
        // the two replays share nothing but the gradient they add to
        cudaEventRecord(fork_ev, st);
        cudaStreamWaitEvent(st_side, fork_ev, 0);
        launch_emit_adj(lc(), ab, st_side);
        cudaEventRecord(join_ev, st_side);
        launch_trace_adj(lc(), ab, st);
        join_side();
        if (cudaGetLastError() != cudaSuccess)
            r = fail(PHX_E_CUDA, "adjoint kernel launch failed");
    }
    in_adjoint = false;
    if (!r)
        r = sync_and_check();
    if (r) {
        adj_live = ADJ_NO_ROUND;
        return r;
    }
    std::vector<double> gd(std::max(np, 1u));
    CK(cudaMemcpy(gd.data(), adj_grad.p, 8 * (size_t)np, cudaMemcpyDeviceToHost));
    for (uint32_t i = 0; i < np; i++)
        grad[i] = (float)gd[i];
    return PHX_OK;
}

} // namespace phx
