// k_adjoint.cu — reverse-mode derivative of the SPPM image with respect to per-material base
// colour and roughness and per-light power: the adjoint of gather_flux (gather_flux.cl:5-78) and of
// the BSDF / direct-lighting weights (shading.h:150-213, bsdfs.h:77-121, light_sampling.h:302-390)
// along camera and photon paths replayed from their RNG seeds.  No counterpart in the reference.
//
// What is differentiated is the frozen-path estimator: every random or discrete choice of the
// forward render stays fixed — paths, BSDF events, microfacet normals, Russian-roulette factors,
// light-selection probabilities, shadow-ray hit lists, gather neighbourhoods, kernel weights,
// radii and SPPM ratios — and only the weights depend on the parameters.  A BSDF bounce with
// frozen directions has weight W(θ0)·f(θ)/f(θ0) (detached sampling), so
//   d log W / d base_c     = 1/base_c (diffuse, transmission; base = material base × texture)
//                          = (1-p)·base_c/(mb_c·F_c) (metal, Schlick F = base + (1-base)·p)
//   d log W / d roughness  = (d log D(h) + d log G1(v) + d log G1(l)) / dα · dα/d roughness,
// with α = roughness² and roughness = clamp(mb_rough × texture, 0.001, 1).  Light power enters
// linearly; photon power is carried unquantised.  The oracle's frozen estimator
// (oracle/phx_frozen.hpp) evaluates exactly this function in double for the finite-difference
// checks.
//
// The image is I = radiance/R + flux.xyz/(π r_R² N) with flux_R = Σ_n c_n Π_{m>=n} ratio_m
// (ratio 1 in a round without photons), so dI/dc_n = K_n = Π_{m>=n} ratio_m / (π r_R² N).
// Per round n of the backward pass (hit points and photons re-created by the ordinary kernels, or still in
// the buffers from the forward pass's last round):
//   k_gather_adj  a = dL/dI·K_n, S = Σ w_k Φ_k over the round's neighbourhood:
//                 dL/dT = a·A/π·S, dL/dA = a·T/π·S, dL/dΦ_k += w_k·a·T·A/π (float atomics)
//   k_trace_adj   replays the camera path and adds, for every term X it produces with adjoint u
//                 (emission and direct light: dL/dI/R; final throughput: dL/dT; base colour: dL/dA),
//                 Σ_c u_c X_c · d log X_c/dθ; the NEE terms come from the shadow wavefront's samples
//   k_nee_adj     the transmissive surfaces those samples' shadow rays crossed
//   k_emit_adj    replays the photon path; at stored photon k, u = dL/dΦ_k ⊙ Φ_k times
//                 d log Φ_k/dθ (the bounces before the store and 1/L of its light)
// Gradients are summed per block in shared memory (float) and then into doubles; with more parameters than a
// block's shared memory holds, every term goes into a double by itself.
#include "dev_shading.cuh"
#include "gather_walk.cuh"
#include "kernels.hpp"

#include <algorithm>

namespace phx {

// ---- gradient accumulation ---------------------------------------------------------------------
// S, the type that sums of terms are held in: float where a block has partial sums in shared memory
// (AdjBufs::block_sums), double where each sum goes straight to the global doubles, whose precision a float
// in between would lose.
template <class S> struct Sum3 {
    S x = 0, y = 0, z = 0;
    Sum3() = default;
    PHX_DI explicit Sum3(float4 v, float s = 1.0f) : x(v.x * (S)s), y(v.y * (S)s), z(v.z * (S)s) {}
    PHX_DI Sum3 &operator+=(const Sum3 &o) {
        x += o.x;
        y += o.y;
        z += o.z;
        return *this;
    }
    PHX_DI bool any() const { return x != 0 || y != 0 || z != 0; }
};

template <class S> struct GradAcc {
    float *sm; // per-block partial sums (S = float)
    double *gl;
    PHX_DI void add(u32 i, S v) const {
        if (v == 0)
            return;
        if constexpr (sizeof(S) == 4)
            atomicAdd(&sm[i], v);
        else
            atomicAdd(&gl[i], v);
    }
    // Four consecutive entries at once.  The lanes that add to the same entries (most of a warp: few
    // materials hold most hits) sum their values by shuffles first: a shared-memory float addition is a
    // compare-and-swap loop, which 32 lanes on one address run 32 times, and a global one serialises as well.
    PHX_DI void add4(u32 o, S a, S b, S c, S d) const {
        const u32 peers = __match_any_sync(__activemask(), o);
        S s0 = 0, s1 = 0, s2 = 0, s3 = 0;
        for (u32 m = peers; m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            s0 += __shfl_sync(peers, a, src);
            s1 += __shfl_sync(peers, b, src);
            s2 += __shfl_sync(peers, c, src);
            s3 += __shfl_sync(peers, d, src);
        }
        if ((threadIdx.x & 31u) == (u32)__ffs(peers) - 1u) {
            add(o, s0);
            add(o + 1, s1);
            add(o + 2, s2);
            add(o + 3, s3);
        }
    }
    // z ⊙ v to three entries
    PHX_DI void add3(u32 o, const Sum3<S> &z, float4 v) const { add4(o, z.x * v.x, z.y * v.y, z.z * v.z, 0); }
};

template <class S> PHX_DI GradAcc<S> grad_begin(const AdjBufs &ab, float *smem) {
    if constexpr (sizeof(S) == 4) {
        for (u32 i = threadIdx.x; i < ab.n_params; i += blockDim.x)
            smem[i] = 0.0f;
        __syncthreads();
    }
    return GradAcc<S>{smem, ab.grad};
}
template <class S> PHX_DI void grad_end(const AdjBufs &ab, const GradAcc<S> &g) {
    if constexpr (sizeof(S) == 4) {
        __syncthreads();
        for (u32 i = threadIdx.x; i < ab.n_params; i += blockDim.x)
            if (g.sm[i] != 0.0f)
                atomicAdd(&ab.grad[i], (double)g.sm[i]);
    }
}

// ---- log-derivatives of the weights ------------------------------------------------------------
PHX_DI float dlog_ndf(float c, float a) { // d log D(c; α) / dα, D = α²/max(π d², EPS) (bsdfs.h:117-121)
    float a2 = a * a;
    float d = c * c * (a2 - 1.0f) + 1.0f;
    if (PI * d * d <= EPS)
        return 2.0f / a;
    return 2.0f / a - 4.0f * a * c * c / d;
}
PHX_DI float dlog_g1(float c, float a) { // d log G1(c; α) / dα (bsdfs.h:77-83); 0 where G1 = 0
    if (c <= 0.0f)
        return 0.0f;
    float a2 = a * a;
    float s = sqrtf(a2 + (1.0f - a2) * c * c);
    return -a * (1.0f - c * c) / (s * (c + s));
}
PHX_DI float4 inv_nonzero(float4 v) {
    return f4(v.x != 0.0f ? 1.0f / v.x : 0.0f, v.y != 0.0f ? 1.0f / v.y : 0.0f, v.z != 0.0f ? 1.0f / v.z : 0.0f,
              0.0f);
}
// dα / d(material roughness) where the clamp is inactive: α = r², r = mb_r·t  =>  2r·t = 2r²/mb_r
PHX_DI float dalpha_drough(float r, float mb_r) {
    return (r > MIN_ROUGHNESS && r < 1.0f && mb_r > 0.0f) ? 2.0f * r * r / mb_r : 0.0f;
}

// d log W of one bounce: per base colour channel of its material, and per material roughness
struct BounceRec {
    u32 mat;
    float db0, db1, db2, dr;
};

PHX_DI BounceRec bounce_dlog(const BsdfSample &bs, float4 h, float4 view, float4 sn, const ShadingContext &ctx,
                             const phx_material &mat, u32 mi) {
    BounceRec r{mi, 0.0f, 0.0f, 0.0f, 0.0f};
    const float4 imb = inv_nonzero(f4(mat.base_color));
    if (bs.event == BSDF_DIFFUSE || bs.event == BSDF_TRANSMIT) {
        r.db0 = imb.x;
        r.db1 = imb.y;
        r.db2 = imb.z;
    } else if (bs.event == BSDF_METALLIC) {
        const float p = pm_powf(1.0f - fabsf(dot(-view, h)), 5.0f);
        const float4 b = ctx.base_color;
        const float fx = b.x + (1.0f - b.x) * p, fy = b.y + (1.0f - b.y) * p, fz = b.z + (1.0f - b.z) * p;
        r.db0 = fx != 0.0f ? (1.0f - p) * b.x * imb.x / fx : 0.0f;
        r.db1 = fy != 0.0f ? (1.0f - p) * b.y * imb.y / fy : 0.0f;
        r.db2 = fz != 0.0f ? (1.0f - p) * b.z * imb.z / fz : 0.0f;
    }
    if (bs.event != BSDF_DIFFUSE) {
        const float a = ctx.roughness * ctx.roughness;
        const float ch = dot(sn, h), cv = fabsf(dot(view, sn));
        const float cl = bs.event == BSDF_TRANSMIT ? fabsf(dot(bs.dir, sn)) : fmaxf(0.0f, dot(bs.dir, sn));
        r.dr = (dlog_ndf(ch, a) + dlog_g1(cv, a) + dlog_g1(cl, a)) * dalpha_drough(ctx.roughness, mat.roughness);
    }
    return r;
}

// Adds Σ_c z_c · d log W_i,c/dθ for every recorded bounce i (z = u ⊙ X of a term X that carries
// the product of those bounce weights).
template <class S> PHX_DI void add_prefix(const GradAcc<S> &acc, const BounceRec *br, u32 nb, const Sum3<S> &z) {
    if (!z.any())
        return;
    const S zs = z.x + z.y + z.z;
    for (u32 i = 0; i < nb; i++) {
        acc.add4(4 * br[i].mat, z.x * br[i].db0, z.y * br[i].db1, z.z * br[i].db2, zs * br[i].dr);
    }
}

// ---- direct lighting with the pieces the adjoint needs -----------------------------------------
struct NeeRec {
    u32 light;          // selected light
    u32 n_occ;          // transmissive occluders on the shadow ray
    u32 occ[MAX_RAY_BOUNCES];
    float dlog_a;       // specular: d log (D G1 G1) / dα
    float4 dlog_f0;     // specular: d log F_c / d f0_c (f0 = base: metal)
};

// shadow_transmittance (light_sampling.h:302-333) recording the transmissive occluders
PHX_DI float4 shadow_tr_rec(const SceneDesc &sc, float4 origin, float4 dir, float dist, u32 *overflow, NeeRec *nr) {
    float4 trans = white4();
    float t_min = EPS, t_max = dist - EPS;
    nr->n_occ = 0;
    for (u32 depth = 0; depth < MAX_RAY_BOUNCES; depth++) {
        Hit h;
        if (!intersect(sc, origin, dir, t_min, t_max, &h, overflow, sc.any_transmissive == 0))
            break;
        u32 mi = tri_mat(sc, h.tri);
        const phx_material &mat = sc.materials[mi];
        if (mat.transmission < EPS)
            return zero4();
        float4 base = f4(mat.base_color);
        if (mat.diff_index != NO_TEXTURE) {
            SurfaceHit s = process_hit(sc, h, origin, dir);
            base *= srgb_to_linear(sample_texture_uv(sc, mi, mat.diff_index, s.uvx, s.uvy, 0));
        }
        if (mat.att_dist > EPS)
            trans *= beer_lambert(f4(mat.att_color), mat.att_dist, h.t - t_min);
        trans *= base * mat.transmission;
        if (dot(trans, trans) < EPS)
            return zero4();
        nr->occ[nr->n_occ++] = mi;
        t_min = h.t + EPS;
    }
    return trans;
}

PHX_DI u32 peek_light(const Rng *rng, const SceneDesc &sc) {
    Rng c = *rng;
    float scale;
    return select_light(&c, sc, &scale);
}

// direct_lighting_diffuse (light_sampling.h:335-353)
PHX_DI float4 nee_diffuse_adj(Rng *rng, const SceneDesc &sc, float4 pos, float4 normal, float4 base, u32 *overflow,
                              NeeRec *nr) {
    nr->light = peek_light(rng, sc);
    nr->n_occ = 0;
    LightFragment f;
    if (!sample_light_fragment(rng, sc, pos, normal, &f))
        return zero4();
    float4 trans = shadow_tr_rec(sc, pos, f.dir, f.dist, overflow, nr);
    return f.radiance * (base / PI) * trans;
}

// direct_lighting_specular (light_sampling.h:355-390); REC: the sample's contribution is known (`known`,
// from the shadow pass), so nothing is traced
template <bool REC>
PHX_DI float4 nee_specular_adj(Rng *rng, const SceneDesc &sc, float4 pos, float4 normal, float4 view, float4 f0,
                               float roughness, u32 *overflow, NeeRec *nr, float4 known) {
    nr->n_occ = 0;
    nr->light = 0;
    float ndv = dot(view, normal);
    if (ndv < EPS)
        return zero4();
    nr->light = peek_light(rng, sc);
    LightFragment f;
    if (!sample_light_fragment(rng, sc, pos, normal, &f))
        return zero4();
    if (f.n_dot_dir < EPS)
        return zero4();
    float alpha = roughness * roughness;
    float4 h = normalize(f.dir + view);
    float ndh = fmaxf(dot(normal, h), 0.0f);
    float g = ggx_ndf(ndh, alpha);
    float4 fr = fresnel4(f0, view, h);
    float sm = smith_g1_ggx(f.n_dot_dir, alpha) * smith_g1_ggx(ndv, alpha);
    float4 spec = f.radiance * g * fr * sm / (4.0f * f.n_dot_dir * ndv);
    if (dot(spec, spec) < EPS * EPS)
        return zero4();
    const float4 v = REC ? known : spec * shadow_tr_rec(sc, pos, f.dir, f.dist, overflow, nr);
    nr->dlog_a = dlog_ndf(ndh, alpha) + dlog_g1(f.n_dot_dir, alpha) + dlog_g1(ndv, alpha);
    const float p = pm_powf(1.0f - fabsf(dot(view, h)), 5.0f);
    nr->dlog_f0 = f4(fr.x != 0.0f ? (1.0f - p) / fr.x : 0.0f, fr.y != 0.0f ? (1.0f - p) / fr.y : 0.0f,
                     fr.z != 0.0f ? (1.0f - p) / fr.z : 0.0f, 0.0f);
    return v;
}

// per-sample derivatives of a NEE term z = u ⊙ X: its light and its transmissive occluders
template <class S>
PHX_DI void add_nee_common(const SceneDesc &sc, const AdjBufs &ab, const GradAcc<S> &acc, const NeeRec &nr,
                           const Sum3<S> &z) {
    if (sc.n_lights > 0)
        acc.add3(4 * ab.n_mat + 3 * nr.light, z, inv_nonzero(f4(sc.lights[nr.light].power)));
    for (u32 i = 0; i < nr.n_occ; i++)
        acc.add3(4 * nr.occ[i], z, inv_nonzero(f4(sc.materials[nr.occ[i]].base_color)));
}

// ---- camera paths (trace_rays.cl:14-169) -------------------------------------------------------
// REC: the round's camera pass left its NEE samples to the shadow wavefront, so every sample's
// contribution is at hand — the diffuse hit point's mean in hp_direct, a specular event's in its sample
// slots — and the replay traces no shadow ray.  Where materials transmit, the occluders a shadow ray
// crossed are needed too: k_nee_adj finds them, one thread per sample, with the pixel's weight left in
// gT.  Otherwise (the one-thread camera kernel, or a specular event that found no free slots) the
// samples are traced here, one after another: 6.2 ms for 512 x 512 pixels of the atrium at 16 samples,
// against 0.72 ms recorded; 1.45 against 0.29 + 0.06 (k_nee_adj) for 97 x 65 pixels through glass at 8.
template <bool REC, class S>
PHX_DI void trace_adj_pixel(const SceneDesc &sc, u32 seed, u32 tid, u32 gpix, const AdjBufs &ab,
                            const GradAcc<S> &acc, u32 *overflow) {
    const float4 ur = ab.g_img[gpix] * ab.inv_rounds; // dL / d(this round's radiance increment)
    const float4 uT = ab.gT[gpix], uA = ab.gA[gpix];
    if (ur.x == 0.0f && ur.y == 0.0f && ur.z == 0.0f && uT.x == 0.0f && uT.y == 0.0f && uT.z == 0.0f &&
        uA.x == 0.0f && uA.y == 0.0f && uA.z == 0.0f)
        return;
    u32 width = sc.width, height = sc.height;
    u32 px = tid % width;
    u32 py = tid / width;
    Rng rng = pcg_seed(seed + tid);
    float4 origin, dir;
    make_ray(sc.camera, px, py, width, height, &rng, &origin, &dir);
    float4 throughput = white4();
    IorStack ior;
    init_ior_stack(&ior, AIR_IOR);
    BounceRec br[MAX_RAY_BOUNCES];
    u32 nb = 0;
    const float inv_ds = 1.0f / (float)sc.direct_samples;
    u32 n_list = 0, at = 0; // REC: the pixel's listed emission terms, and the next one to look at
    if constexpr (REC) {
        n_list = ab.tr.def_cnt[gpix] & 0xffu;
        ab.gT[gpix] = zero4(); // read above; the diffuse samples' weight below
    }
    for (i32 depth = 0; depth < (i32)MAX_RAY_BOUNCES; depth++) {
        Hit h;
        bool hit = intersect(sc, origin, dir, EPS, INF, &h, overflow);
        if (!hit) {
            if (sc.has_env)
                add_prefix(acc, br, nb, Sum3<S>(ur * throughput * sample_envmap(sc, dir)));
            break;
        }
        const phx_material mat = sc.materials[tri_mat(sc, h.tri)];
        SurfaceHit sh = process_hit(sc, h, origin, dir, mat_textured(mat));
        float cur = current_ior(&ior);
        if (cur != AIR_IOR && mat.thickness > EPS && mat.att_dist > EPS)
            throughput *= beer_lambert(f4(mat.att_color), mat.att_dist, sh.t);
        float4 tangent = zero4(), bitangent = zero4(); // the frame only serves a normal map
        if (mat.norm_index != NO_TEXTURE)
            hit_frame(sc, h, sh, &tangent, &bitangent);
        ShadingContext ctx = evaluate_material(sc, mat, sh.mat_index, sh.uvx, sh.uvy, sh.normal, tangent, bitangent);
        add_prefix(acc, br, nb, Sum3<S>(ur * throughput * ctx.emissive));
        float4 view = -dir;
        float4 hm; // the microfacet normal
        BsdfSample bs = sample_bsdf_h(&rng, ctx, ctx.shading_normal, sh.normal, view, &ior, sh.front_face, &hm);
        const u32 mo = 4 * sh.mat_index;
        const float4 imb = inv_nonzero(f4(mat.base_color));
        if (bs.event == BSDF_DIFFUSE) {
            // direct = T·occlusion·mean_s NEE_s, NEE_s = L_s·base/π·trans_s
            const float4 w = ur * throughput * (ctx.occlusion * inv_ds);
            Sum3<S> zsum;
            if constexpr (REC) {
                const float4 *val = ab.tr.nee_val + sc.nee_base + (size_t)(gpix - sc.pixel_base) * sc.direct_samples;
                if constexpr (sizeof(S) == 4)
                    zsum = Sum3<S>(ur * ab.tr.direct[gpix]); // the pass's own float mean of the samples
                else
                    for (u32 d = 0; d < sc.direct_samples; d++)
                        zsum += Sum3<S>(w * val[d]);
                if (sc.n_lights == 1) {
                    acc.add3(4 * ab.n_mat, zsum, inv_nonzero(f4(sc.lights[0].power)));
                } else {
                    for (u32 d = 0; d < sc.direct_samples; d++) { // which light each sample chose
                        NeeRec nr;
                        nr.n_occ = 0;
                        nr.light = peek_light(&rng, sc);
                        if (sc.light_draws == LIGHT_DRAWS_VARY) {
                            LightFragment f;
                            sample_light_fragment(&rng, sc, sh.position, ctx.shading_normal, &f);
                        } else {
                            rng = rng_advance(rng, sc.light_draws);
                        }
                        const Sum3<S> z(w * val[d]);
                        if (z.any())
                            add_nee_common(sc, ab, acc, nr, z);
                    }
                }
                ab.gT[gpix] = w;
            } else {
                for (u32 d = 0; d < sc.direct_samples; d++) {
                    NeeRec nr;
                    float4 v =
                        nee_diffuse_adj(&rng, sc, sh.position, ctx.shading_normal, ctx.base_color, overflow, &nr);
                    const Sum3<S> z(w * v);
                    if (!z.any())
                        continue;
                    zsum += z;
                    add_nee_common(sc, ab, acc, nr, z);
                }
            }
            Sum3<S> zp = zsum; // direct light, and the hit point's throughput
            zp += Sum3<S>(uT * throughput);
            add_prefix(acc, br, nb, zp);
            zsum += Sum3<S>(uA * ctx.base_color); // the hit point's base colour (mb × texture)
            acc.add3(mo, zsum, imb);
            break;
        }
        if (bs.event == BSDF_METALLIC || bs.event == BSDF_FRESNEL) {
            float4 f0 = ctx.base_color;
            if (bs.event == BSDF_FRESNEL) {
                float ratio = (cur - ctx.ior) / (cur + ctx.ior);
                float r0 = ratio * ratio;
                f0 = f4(r0, r0, r0, 0.0f);
            }
            const float dadr = dalpha_drough(ctx.roughness, mat.roughness);
            const float4 w = ur * throughput * inv_ds;
            Sum3<S> zsum, gb; // gb, gr: d/d base colour (metal), d/d roughness
            S gr = 0;
            u32 slots = DEF_KNOWN;
            if constexpr (REC) // the next event of the pixel's list (events past its slots are not in it)
                while (at < n_list && slots == DEF_KNOWN)
                    slots = ab.tr.def_tag[(size_t)gpix * DEF_MAX + at++];
            auto add_sample = [&](const NeeRec &nr, const Sum3<S> &z) {
                if (!z.any())
                    return;
                zsum += z;
                add_nee_common(sc, ab, acc, nr, z);
                gr += (z.x + z.y + z.z) * nr.dlog_a * dadr;
                if (bs.event == BSDF_METALLIC) { // f0 = base = mb × texture
                    const float4 b = ctx.base_color;
                    gb.x += z.x * nr.dlog_f0.x * b.x * imb.x;
                    gb.y += z.y * nr.dlog_f0.y * b.y * imb.y;
                    gb.z += z.z * nr.dlog_f0.z * b.z * imb.z;
                }
            };
            if (REC && slots != DEF_KNOWN) {
                // one light that takes one draw: its samples are all the same
                const u32 same = ab.same_samples ? sc.direct_samples : 1u;
                for (u32 d = 0; d < sc.direct_samples; d += same) {
                    NeeRec nr;
                    const Rng before = rng;
                    const float4 v = nee_specular_adj<true>(&rng, sc, sh.position, ctx.shading_normal, view, f0,
                                                            ctx.roughness, overflow, &nr, ab.tr.spec_val[slots + d]);
                    if (same > 1 && rng.state != before.state)
                        rng = rng_advance(before, same * sc.light_draws);
                    add_sample(nr, Sum3<S>(w * v, (float)same));
                }
            } else {
                for (u32 d = 0; d < sc.direct_samples; d++) {
                    NeeRec nr;
                    float4 v = nee_specular_adj<false>(&rng, sc, sh.position, ctx.shading_normal, view, f0,
                                                       ctx.roughness, overflow, &nr, zero4());
                    add_sample(nr, Sum3<S>(w * v));
                }
            }
            acc.add4(mo, gb.x, gb.y, gb.z, gr);
            add_prefix(acc, br, nb, zsum);
        }
        br[nb++] = bounce_dlog(bs, hm, view, ctx.shading_normal, ctx, mat, sh.mat_index);
        throughput *= bs.throughput;
        if ((u32)depth >= RR_MIN_RAY_DEPTH) {
            float q = fmaxf(throughput.x, fmaxf(throughput.y, throughput.z));
            q = clampf(q, RR_MIN_Q, RR_MAX_Q);
            if (random_float(&rng) > q)
                break;
            throughput *= 1.0f / q;
        }
        float4 side = (dot(bs.dir, sh.normal) > 0.0f) ? sh.normal : -sh.normal;
        origin = sh.position + bs.dir * EPS + side * EPS;
        dir = bs.dir;
    }
}

template <bool REC, class S>
__global__ void __launch_bounds__(128) k_trace_adj(LaunchCtx lc, AdjBufs ab) {
    extern __shared__ float s_grad[];
    const GradAcc<S> acc = grad_begin<S>(ab, s_grad);
    u32 gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid < lc.total_pixels) {
        const SceneDesc &sc = lc.scenes[0];
        u32 ovf = 0;
        trace_adj_pixel<REC, S>(sc, __ldg(&lc.seeds[0]), gid, gid, ab, acc, &ovf);
        if (ovf)
            atomicAdd(lc.overflow, ovf);
    }
    grad_end(ab, acc);
}

// Occluders of the recorded NEE samples (scenes with transmissive materials): one thread per sample slot,
// the diffuse hit points' first, then the specular events'.  A sample that contributes is drawn again
// as the shadow pass drew it and its ray traced once more for the surfaces it crossed.
template <class S> __global__ void __launch_bounds__(128) k_nee_adj(LaunchCtx lc, AdjBufs ab, u32 nee_blocks) {
    extern __shared__ float s_grad[];
    const GradAcc<S> acc = grad_begin<S>(ab, s_grad);
    const SceneDesc &sc = lc.scenes[0];
    const TraceOut &out = ab.tr;
    const u32 ds = sc.direct_samples, same = ab.same_samples ? ds : 1u;
    u32 ovf = 0;
    auto crossed = [&](float4 org, float4 dir, float dist, const Sum3<S> &z) {
        NeeRec nr;
        shadow_tr_rec(sc, org, dir, dist, &ovf, &nr);
        for (u32 i = 0; i < nr.n_occ; i++)
            acc.add3(4 * nr.occ[i], z, inv_nonzero(f4(sc.materials[nr.occ[i]].base_color)));
    };
    if (blockIdx.x < nee_blocks) {
        const u32 t = (blockIdx.x * blockDim.x + threadIdx.x) * same;
        if (t < lc.total_nee && out.emission[t / ds].w == 1.0f) {
            const u32 gpix = t / ds;
            const Sum3<S> z(ab.gT[gpix] * out.nee_val[t], (float)same);
            if (z.any()) {
                if (sc.light_draws != LIGHT_DRAWS_VARY) {
                    Rng rng;
                    rng.state = out.stash_rng[gpix];
                    rng = rng_advance(rng, (t - gpix * ds) * sc.light_draws);
                    LightFragment f;
                    if (light_fragment(&rng, sc, out.pos[gpix], out.stash_sn[gpix], &f))
                        crossed(out.pos[gpix], f.dir, f.dist, z);
                } else {
                    const float4 ray = out.nee_ray[t];
                    crossed(out.pos[gpix], f4(ray.x, ray.y, ray.z, 0.0f), ray.w, z);
                }
            }
        }
    } else {
        const u32 n = min(*out.spec_next, out.spec_cap), stride = (gridDim.x - nee_blocks) * blockDim.x;
        for (u32 e = (blockIdx.x - nee_blocks) * blockDim.x + threadIdx.x; (u64)e * same < n; e += stride) {
            const u32 g = e * same, base = g / ds * ds; // events claim ds slots each
            const u32 gpix = out.spec_pix[g], listed = out.def_cnt[gpix] & 0xffu;
            Sum3<S> z;
            for (u32 k = 0; k < listed; k++)
                if (out.def_tag[(size_t)gpix * DEF_MAX + k] == base)
                    z = Sum3<S>(ab.g_img[gpix] * ab.inv_rounds * out.def_val[(size_t)gpix * DEF_MAX + k] *
                                    (1.0f / (float)ds) * out.spec_val[g],
                                (float)same);
            if (!z.any())
                continue;
            const float4 hdr = out.spec_ray[g];
            if (spec_drawn_in_shadow(sc)) {
                Rng rng;
                rng.state = __float_as_uint(hdr.z);
                rng = rng_advance(rng, (g - base) * sc.light_draws);
                LightFragment f;
                if (light_fragment(&rng, sc, out.spec_org[base], out.spec_org[base + 1], &f))
                    crossed(out.spec_org[base], f.dir, f.dist, z);
            } else {
                crossed(out.spec_org[g], f4(hdr.x, hdr.y, hdr.z, 0.0f), hdr.w, z);
            }
        }
    }
    if (ovf)
        atomicAdd(lc.overflow, ovf);
    grad_end(ab, acc);
}

// ---- photon paths (emit_photons.cl:12-114) -----------------------------------------------------
constexpr u32 MAX_PHOTON_BOUNCES = 32;

template <class S>
PHX_DI void emit_adj_path(const SceneDesc &sc, u32 seed, u32 tid, const AdjBufs &ab, const GradAcc<S> &acc,
                          u32 *overflow) {
    u32 k = ab.offsets[tid];
    const u32 n_stored = ab.offsets[tid + 1] - k;
    Rng rng = pcg_seed(seed + tid);
    const u32 li = peek_light(&rng, sc);
    float4 origin, dir, power;
    sample_light(&rng, sc, &origin, &dir, &power);
    const float4 il = sc.n_lights > 0 ? inv_nonzero(f4(sc.lights[li].power)) : zero4();
    const u32 lo = 4 * ab.n_mat + 3 * li;
    IorStack ior;
    init_ior_stack(&ior, AIR_IOR);
    float4 throughput = f4(1.0f, 1.0f, 1.0f, 0.0f);
    BounceRec br[MAX_PHOTON_BOUNCES];
    float4 stored[MAX_PHOTON_BOUNCES + 1]; // dL/dΦ ⊙ Φ of the photon stored after so many bounces
    stored[0] = zero4();
    u32 nb = 0, seen = 0;
    for (u32 depth = 0; depth < sc.max_bounces && seen < n_stored; depth++) {
        Hit h;
        bool hit = intersect(sc, origin, dir, EPS, INF, &h, overflow);
        if (!hit)
            break;
        const phx_material mat = sc.materials[tri_mat(sc, h.tri)];
        SurfaceHit sh = process_hit(sc, h, origin, dir, mat_textured(mat));
        float cur = current_ior(&ior);
        if (cur != AIR_IOR && mat.thickness > EPS && mat.att_dist > EPS) {
            float4 vol = beer_lambert(f4(mat.att_color), mat.att_dist, sh.t);
            power *= vol;
            throughput *= vol;
        }
        float4 tangent = zero4(), bitangent = zero4(); // the frame only serves a normal map
        if (mat.norm_index != NO_TEXTURE)
            hit_frame(sc, h, sh, &tangent, &bitangent);
        ShadingContext ctx = evaluate_material(sc, mat, sh.mat_index, sh.uvx, sh.uvy, sh.normal, tangent, bitangent);
        if (depth >= RR_MIN_PHOTON_DEPTH) {
            float q = fmaxf(throughput.x, fmaxf(throughput.y, throughput.z));
            q = clampf(q, RR_MIN_Q, RR_MAX_Q);
            if (random_float(&rng) > q)
                break;
            float inv_q = 1.0f / q;
            throughput *= inv_q;
            power *= inv_q;
        }
        float4 view = -dir;
        float4 hm; // the microfacet normal
        BsdfSample bs = sample_bsdf_h(&rng, ctx, ctx.shading_normal, sh.normal, view, &ior, sh.front_face, &hm);
        stored[nb] = zero4();
        if (bs.event == BSDF_DIFFUSE && dot(dir, sh.normal) < 0.0f) {
            stored[nb] = ab.gphi[k] * power; // dL/dΦ ⊙ Φ of this stored photon
            k++;
            seen++;
            if (seen == n_stored) { // no photon is stored later: this bounce weighs nothing
                nb++;
                break;
            }
        }
        br[nb++] = bounce_dlog(bs, hm, view, ctx.shading_normal, ctx, mat, sh.mat_index);
        power *= bs.throughput;
        throughput *= bs.throughput;
        float4 side = (dot(bs.dir, sh.normal) > 0.0f) ? sh.normal : -sh.normal;
        origin = sh.position + bs.dir * EPS + side * EPS;
        dir = bs.dir;
    }
    // bounce i weighs every photon stored after it; the light weighs all of them: one sum per bounce, not
    // one per bounce and photon (atrium, 2^20 paths: 1.60 -> 1.06 ms with the shuffled sums)
    Sum3<S> z;
    for (u32 i = nb; i-- > 0;) {
        if (i + 1 < nb && z.any())
            acc.add4(4 * br[i].mat, z.x * br[i].db0, z.y * br[i].db1, z.z * br[i].db2, (z.x + z.y + z.z) * br[i].dr);
        z += Sum3<S>(stored[i]);
    }
    acc.add3(lo, z, il);
}

// The paths that stored a photon (one in six of the atrium's), so that every lane of k_emit_adj has one to
// replay: 1.06 -> 0.47 + 0.03 ms for the 2^20 paths of the 512 x 512 atrium.
__global__ void __launch_bounds__(256) k_adj_paths(LaunchCtx lc, AdjBufs ab) {
    const u32 gid = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const bool stored = gid < lc.total_emit && ab.offsets[gid + 1] != ab.offsets[gid];
    const u32 m = __ballot_sync(0xffffffffu, stored);
    u32 base = 0;
    if (lane == 0 && m)
        base = atomicAdd(ab.n_paths, (u32)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (stored)
        ab.paths[base + __popc(m & ((1u << lane) - 1u))] = gid;
}

template <class S> __global__ void __launch_bounds__(128) k_emit_adj(LaunchCtx lc, AdjBufs ab) {
    extern __shared__ float s_grad[];
    const GradAcc<S> acc = grad_begin<S>(ab, s_grad);
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < *ab.n_paths) {
        const SceneDesc &sc = lc.scenes[0];
        u32 ovf = 0;
        emit_adj_path(sc, __ldg(&lc.seeds[0]), ab.paths[i], ab, acc, &ovf);
        if (ovf)
            atomicAdd(lc.overflow, ovf);
    }
    grad_end(ab, acc);
}

// ---- gather adjoint (gather_flux.cl:5-78, photon_hash.h:56-103) --------------------------------
// Bound by the photon records' latency and, before the walk of the forward gather was shared, by the few lanes
// that ran a pair's weight, loads and reduction while the others waited: with the queue they run together.
// A round's 16-byte reductions stay, one a pair.  One-round step of the 512 x 512 atrium 5.38 -> 4.79 ms,
// two-round step of a 97 x 65 caustic box 2.69 -> 2.48.  8 blocks an SM and two pairs in flight: a pair holds
// a record index more than the forward gather's.
constexpr u32 GA_BATCH = 2;
__global__ void __launch_bounds__(128, 8) k_gather_adj(LaunchCtx lc, GatherBufs g, AdjBufs ab) {
    __shared__ u32 q_k[GQ_CAP][128];
    __shared__ float q_d[GQ_CAP][128];
    const u32 tid = threadIdx.x;
    u32 gpix = blockIdx.x * blockDim.x + tid;
    const SceneDesc &sc = lc.scenes[0];
    bool gathering = false;
    float4 a = zero4(), pos = zero4(), nrm = zero4(), pa = zero4(), S = zero4();
    float r_sq = 0.0f;
    NearCells nc;
    if (gpix < lc.total_pixels) {
        if (g.order) // any round's order will do: it only decides which pixels share a warp
            gpix = __ldg(&g.order[gpix]);
        a = ab.g_img[gpix] * ab.kscale[gpix];
        gathering = !(g.hp_emission[gpix].w == 0.0f || (a.x == 0.0f && a.y == 0.0f && a.z == 0.0f));
        if (!gathering) {
            ab.gT[gpix] = zero4();
            ab.gA[gpix] = zero4();
        }
    }
    if (gathering) {
        r_sq = ab.r2[gpix];
        pos = g.hp_pos[gpix];
        nrm = g.hp_normal[gpix];
        pa = a * g.hp_throughput[gpix] * (g.hp_base_color[gpix] / PI); // dL/dΦ_k = w_k · pa
        nc = near_cells(pos, r_sq, sc.grid);
    }
    const KernelWeight weight(r_sq);
    walk_photons(g, g.cell_start + sc.cell_base, sc.grid.g, nc, pos, r_sq, q_k, q_d, tid, [&](u32 cnt) {
        for (u32 e = 0; __any_sync(0xffffffffu, e < cnt); e += GA_BATCH) {
            if (e >= cnt)
                continue;
            float4 pd[GA_BATCH], pw[GA_BATCH];
            u32 c[GA_BATCH];
#pragma unroll
            for (u32 u = 0; u < GA_BATCH; u++) {
                const u32 k = q_k[min(e + u, cnt - 1u)][tid];
                c[u] = __ldg(&ab.perm[k]);
                pd[u] = __ldg(&g.s_dir[k]); // decode_oct(p.w)
            }
#pragma unroll
            for (u32 u = 0; u < GA_BATCH; u++)
                pw[u] = __ldg(&ab.ph_pow[c[u]]);
#pragma unroll
            for (u32 u = 0; u < GA_BATCH; u++) {
                if (e + u < cnt && !(dot(pd[u], nrm) > 0.0f)) {
                    const float w = weight(q_d[e + u][tid]);
                    S += w * pw[u];
                    atomicAdd(&ab.gphi[c[u]], f4(w * pa.x, w * pa.y, w * pa.z, 0.0f)); // one 16-byte reduction
                }
            }
        }
    });
    if (!gathering)
        return;
    ab.gT[gpix] = a * (g.hp_base_color[gpix] / PI) * S;
    ab.gA[gpix] = a * (g.hp_throughput[gpix] / PI) * S;
}

// ---- small kernels -------------------------------------------------------------------------------
// unquantised power of the canonical photons (the compaction of k_compact for the power slots)
__global__ void __launch_bounds__(256) k_compact_pow(LaunchCtx lc, const float4 *slot_pow, const u32 *counts,
                                                     const u32 *offsets, float4 *ph_pow) {
    u32 gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= lc.total_emit)
        return;
    const SceneDesc &sc = lc.scenes[0];
    const u32 c = counts[gid], off = offsets[gid];
    u64 slot = sc.slot_base + gid;
    for (u32 j = 0; j < c; j++, slot += sc.n_emit)
        ph_pow[off + j] = slot_pow[slot];
}

// K_n = Π_{m>=n} ratio_m / (π r_R² N) per pixel, rounds stored round-major
__global__ void __launch_bounds__(256) k_adj_scale(const float *ratio, float *kscale, const float4 *flux, u32 n_pix,
                                                   u32 rounds, float inv_n) {
    u32 p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pix)
        return;
    const float area = PI * flux[p].w;
    float k = area > 0.0f ? inv_n / area : 0.0f;
    for (u32 n = rounds; n-- > 0;) {
        k *= ratio[(size_t)n * n_pix + p];
        kscale[(size_t)n * n_pix + p] = k;
    }
}

__global__ void __launch_bounds__(256) k_adj_begin(const float *g3, float4 *g4, u32 n_pix) {
    const u32 p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n_pix)
        g4[p] = f4(g3[3 * (size_t)p], g3[3 * (size_t)p + 1], g3[3 * (size_t)p + 2], 0.0f);
}
__global__ void __launch_bounds__(256) k_adj_clear(float4 *gphi, const u32 *n, u64 n_max) {
    const u64 m = min((u64)*n, n_max);
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (u64)gridDim.x * blockDim.x)
        gphi[i] = zero4();
}

// linear image radiance/R + flux/(π r² N) (output.cpp:62-76 before the display transform)
__global__ void __launch_bounds__(256) k_adj_image(const float4 *flux, const float4 *radiance, u32 n_pix,
                                                   float inv_rounds, float inv_n, float *img) {
    u32 p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pix)
        return;
    const float4 f = flux[p], r = radiance[p];
    const float area = PI * f.w;
    const float per = area > 0.0f ? inv_n / area : 0.0f;
    img[3 * (size_t)p + 0] = r.x * inv_rounds + f.x * per;
    img[3 * (size_t)p + 1] = r.y * inv_rounds + f.y * per;
    img[3 * (size_t)p + 2] = r.z * inv_rounds + f.z * per;
}

static size_t grad_smem(const AdjBufs &ab) { return ab.block_sums ? 4 * (size_t)ab.n_params : 0; }

template <class S> static void launch_trace_adj_s(const LaunchCtx &lc, const AdjBufs &ab, cudaStream_t st) {
    const u32 grid = (lc.total_pixels + 127) / 128;
    if (!ab.tr.def_cnt) {
        k_trace_adj<false, S><<<grid, 128, grad_smem(ab), st>>>(lc, ab);
        return;
    }
    k_trace_adj<true, S><<<grid, 128, grad_smem(ab), st>>>(lc, ab);
    if (ab.occluders) {
        const u32 nee_blocks = (lc.total_nee / (ab.same_samples ? ab.same_samples : 1u) + 127) / 128;
        k_nee_adj<S><<<nee_blocks + (u32)g_sm_count * 4u, 128, grad_smem(ab), st>>>(lc, ab, nee_blocks);
    }
}
void launch_trace_adj(const LaunchCtx &lc, const AdjBufs &ab, cudaStream_t st) {
    if (!lc.total_pixels)
        return;
    if (ab.block_sums)
        launch_trace_adj_s<float>(lc, ab, st);
    else
        launch_trace_adj_s<double>(lc, ab, st);
}
void launch_emit_adj(const LaunchCtx &lc, const AdjBufs &ab, cudaStream_t st) {
    if (!lc.total_emit)
        return;
    cudaMemsetAsync(ab.n_paths, 0, sizeof(u32), st);
    k_adj_paths<<<(lc.total_emit + 255) / 256, 256, 0, st>>>(lc, ab);
    const u32 grid = (lc.total_emit + 127) / 128;
    if (ab.block_sums)
        k_emit_adj<float><<<grid, 128, grad_smem(ab), st>>>(lc, ab);
    else
        k_emit_adj<double><<<grid, 128, 0, st>>>(lc, ab);
}
void launch_gather_adj(const LaunchCtx &lc, const GatherBufs &g, const AdjBufs &ab, cudaStream_t st) {
    if (lc.total_pixels)
        k_gather_adj<<<(lc.total_pixels + 127) / 128, 128, 0, st>>>(lc, g, ab);
}
void launch_compact_pow(const LaunchCtx &lc, const float4 *slot_pow, const u32 *counts, const u32 *offsets,
                        float4 *ph_pow, cudaStream_t st) {
    if (lc.total_emit)
        k_compact_pow<<<(lc.total_emit + 255) / 256, 256, 0, st>>>(lc, slot_pow, counts, offsets, ph_pow);
}
void launch_adj_begin(const float *g3, float4 *g4, u32 n_pix, cudaStream_t st) {
    if (n_pix)
        k_adj_begin<<<(n_pix + 255) / 256, 256, 0, st>>>(g3, g4, n_pix);
}
void launch_adj_clear(float4 *gphi, const u32 *n, u64 n_max, cudaStream_t st) {
    if (n_max)
        k_adj_clear<<<(unsigned)std::min<u64>((n_max + 255) / 256, (u64)g_sm_count * 8), 256, 0, st>>>(gphi, n, n_max);
}
void launch_adj_scale(const float *ratio, float *kscale, const float4 *flux, u32 n_pix, u32 rounds, float inv_n,
                      cudaStream_t st) {
    if (n_pix)
        k_adj_scale<<<(n_pix + 255) / 256, 256, 0, st>>>(ratio, kscale, flux, n_pix, rounds, inv_n);
}
void launch_adj_image(const float4 *flux, const float4 *radiance, u32 n_pix, float inv_rounds, float inv_n, float *img,
                      cudaStream_t st) {
    if (n_pix)
        k_adj_image<<<(n_pix + 255) / 256, 256, 0, st>>>(flux, radiance, n_pix, inv_rounds, inv_n, img);
}

} // namespace phx
