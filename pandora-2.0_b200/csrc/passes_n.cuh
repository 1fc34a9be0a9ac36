// passes_n.cuh -- the launchers of the five passes for one transform length N (host
// code), instantiated per group of lengths by the passes_n*.cu files.
#pragma once
#include "passes_kernels.cuh"

namespace pd {

template <int N, class T, int LPW = XCfg<N, T>::lpw> static size_t smem_kx() {
    return sizeof(typename Cplx<T>::type) * (size_t)LPW * XCfg<N, T>::template ls<LPW>();
}

// CTAs of `kernel` resident on the whole device at once.
template <typename K> static long long resident_ctas(K kernel, int threads, size_t smem) {
    int dev = 0, nsm = 1, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess || per < 1) {
        cudaGetLastError();
        per = 1;
    }
    return (long long)nsm * per;
}

template <typename K> static cudaError_t set_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Launches `kernel`, with `pdl` as a programmatic dependent of the kernel before it in the
// stream: its CTAs may be set up once that kernel's have ended (no kernel triggers earlier), and
// wait at grid_wait() until its writes are visible.
template <class... KA, class... A>
static void launch_after(bool pdl, void (*kernel)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);   // the callers read cudaGetLastError
}

#define PD_CAP(S) std::decay_t<decltype(S)>::cap

// Dynamic shared memory limits of the kernels of length N that the geometry uses, for
// member sets of CAP.
template <int N, class T, int CAP> static cudaError_t configure_cap(const Geo& g) {
    cudaError_t e = cudaSuccess;
    // the K1 that zpass_inv_n launches for each form: staged, or element-wise (also for a cubic
    // grid where the length has that form)
    auto k1 = [&](auto form) {
        constexpr int FORM = decltype(form)::value;
        if (e) return;
        if constexpr (staged_len<N, T, FORM>()) {
            e = set_smem(k_zpass_inv_staged<N, FORM, T, CAP>, SCfg<N, T>::smem);
        } else {
            e = set_smem(k_zpass_inv<N, FORM, T, CAP>, TCfg<N>::template smem<T>());
            if constexpr (cube_len<N, T>())
                if (!e && is_cube(g, N)) e = set_smem(k_zpass_inv<N, FORM, T, CAP, N>, TCfg<N>::template smem<T>());
        }
    };
    if (g.nz == N) {
        k1(std::integral_constant<int, 0>{});
        k1(std::integral_constant<int, 1>{});
        k1(std::integral_constant<int, 2>{});
        k1(std::integral_constant<int, 3>{});
        if (e) return e;
        if ((e = set_smem(k_zpass_fwd<N, T, CAP>, TCfg<N, 2>::template smem<T>()))) return e;
    }
    if constexpr (cube_len<N, T>()) {
        if (is_cube(g, N)) {
            if ((e = set_smem(k_ypass_inv<N, T, CAP, N>, TCfg<N, 1>::template smem<T>()))) return e;
            if ((e = set_smem(k_ypass_fwd<N, T, CAP, N>, TCfg<N, 1>::template smem<T>()))) return e;
        }
    }
    if (g.ny == N) {
        if ((e = set_smem(k_ypass_inv<N, T, CAP>, TCfg<N, 1>::template smem<T>()))) return e;
        if ((e = set_smem(k_ypass_fwd<N, T, CAP>, TCfg<N, 1>::template smem<T>()))) return e;
    }
    if (g.nx == N) {
        if constexpr (xlpw_len<N>()) {   // at most 20 KB per warp: no opt-in needed beyond this
            if ((e = set_smem(k_xpass<N, T, CAP, false, 1>, smem_kx<N, T, 1>()))) return e;
            if ((e = set_smem(k_xpass<N, T, CAP, false, 2>, smem_kx<N, T, 2>()))) return e;
            if ((e = set_smem(k_xpass<N, T, CAP, false, 4>, smem_kx<N, T, 4>()))) return e;
        } else {
            constexpr int LPW = XCfg<N, T>::lpw;
            if ((e = set_smem(k_xpass<N, T, CAP, false, LPW>, smem_kx<N, T>()))) return e;
        }
        if (g.rconv && (e = set_smem(k_xpass_conv<N, T, CAP>, ConvCfg<N, T>::smem))) return e;
    }
    return cudaSuccess;
}

template <int N, class T> cudaError_t configure_n(const Geo& g) {
    static_assert(N <= kMaxLength, "mode_row covers the planes of lengths up to kMaxLength");
    cudaError_t e;
    if constexpr (std::is_same<T, double>::value && ZStage<N>::enabled) {
        if (g.nz == N) {
            if ((e = set_smem(k_zpass_inv_tma<N, 0>, ZStage<N>::smem))) return e;
            if ((e = set_smem(k_zpass_inv_tma<N, 1>, ZStage<N>::smem))) return e;
            if ((e = set_smem(k_zpass_inv_tma<N, 2>, ZStage<N>::smem))) return e;
            if ((e = set_smem(k_zpass_inv_tma<N, 3>, ZStage<N>::smem))) return e;
        }
    }
    if ((e = configure_cap<N, T, 1>(g))) return e;
    if constexpr (batch_len<N>()) {
        if ((e = configure_cap<N, T, kBatchChunk>(g))) return e;
    }
    return cudaSuccess;
}

// K1 (z length N): the tensor-copy kernel for a single FP64 simulation with tensor maps, else the
// copy-staged kernel (staged_len) or the element-wise kernel of the flow's form.
template <int N, class T>
cudaError_t zpass_inv_n(const Geo& g, const Member<T>* M, int B, int stage, cudaStream_t st, const ZMaps* maps, bool pdl) {
    if constexpr (std::is_same<T, double>::value && ZStage<N>::enabled) {
        if (maps && B == 1) {
            MemberSet<double, 1> one;
            one.m[0] = M[0];
            const dim3 grid((unsigned)(g.nkip / ZStage<N>::lines), g.nkj);
            constexpr int NT = ZStage<N>::nt;
            constexpr size_t sm = ZStage<N>::smem;
            if (!g.shear) launch_after(pdl, k_zpass_inv_tma<N, 0>, grid, NT, sm, st, one, *maps, stage);
            else if (!g.rrot) launch_after(pdl, k_zpass_inv_tma<N, 1>, grid, NT, sm, st, one, *maps, stage);
            else if (!g.rconv) launch_after(pdl, k_zpass_inv_tma<N, 2>, grid, NT, sm, st, one, *maps, stage);
            else launch_after(pdl, k_zpass_inv_tma<N, 3>, grid, NT, sm, st, one, *maps, stage);
            return cudaGetLastError();
        }
    }
    return for_member_sets(M, B, [&](const auto& ms, int nb) {
        constexpr int CAP = PD_CAP(ms);
        if constexpr (CAP == 1 || batch_len<N>()) {
            const dim3 grid(pass_fields(g) * nb, TCfg<N>::template tiles<T>(g), g.nkj);
            constexpr int NT = TCfg<N>::template nt<T>();
            const size_t sm = TCfg<N>::template smem<T>();
            auto go = [&](auto form, auto cn) {
                constexpr int FORM = decltype(form)::value, CN = decltype(cn)::value;
                if constexpr (staged_len<N, T, FORM>()) {
                    using S = SCfg<N, T>;
                    auto kern = k_zpass_inv_staged<N, FORM, T, CAP>;
                    const long long pf = CAP == 1 ? resident_ctas(kern, S::nt, S::smem) : 0;
                    launch_after(pdl, kern, dim3((unsigned)(g.nkip / S::lines), g.nkj, nb), S::nt, S::smem, st, ms, stage, pf);
                } else {
                    auto kern = k_zpass_inv<N, FORM, T, CAP, CN>;
                    const long long pf = CAP == 1 ? resident_ctas(kern, NT, sm) : 0;
                    launch_after(pdl, kern, grid, NT, sm, st, ms, stage, pf);
                }
            };
            auto form = [&](auto cn) {
                if (!g.shear) go(std::integral_constant<int, 0>{}, cn);
                else if (!g.rrot) go(std::integral_constant<int, 1>{}, cn);
                else if (!g.rconv) go(std::integral_constant<int, 2>{}, cn);
                else go(std::integral_constant<int, 3>{}, cn);
            };
            if constexpr (cube_len<N, T>()) {
                if (is_cube(g, N)) { form(std::integral_constant<int, N>{}); return; }
            }
            form(std::integral_constant<int, 0>{});
        }
    });
}

template <int N, class T> cudaError_t ypass_inv_n(const Geo& g, const Member<T>* M, int B, cudaStream_t st, bool pdl) {
    return for_member_sets(M, B, [&](const auto& ms, int nb) {
        constexpr int CAP = PD_CAP(ms);
        if constexpr (CAP == 1 || batch_len<N>()) {
            const dim3 grid(TCfg<N, 1>::template tiles<T>(g), g.nz, pass_fields(g) * nb);
            constexpr int NT = TCfg<N, 1>::template nt<T>();
            constexpr size_t sm = TCfg<N, 1>::template smem<T>();
            if constexpr (cube_len<N, T>()) {
                if (is_cube(g, N)) { launch_after(pdl, k_ypass_inv<N, T, CAP, N>, grid, NT, sm, st, ms, pass_fields(g)); return; }
            }
            launch_after(pdl, k_ypass_inv<N, T, CAP>, grid, NT, sm, st, ms, pass_fields(g));
        }
    });
}

template <int N, class T>
cudaError_t xpass_n(const Geo& g, const Member<T>* M, int B, int want_phys, int want_cfl, cudaStream_t st, bool pdl) {
    const long long lines = (long long)g.ny * g.nz;
    return for_member_sets(M, B, [&](const auto& ms, int nb) {
        constexpr int CAP = PD_CAP(ms);
        if constexpr (CAP == 1 || batch_len<N>()) {
            if (g.rconv) {   // R-conv: its own x pass
                auto kern = k_xpass_conv<N, T, CAP>;
                const long long pf = CAP == 1 ? resident_ctas(kern, 32, ConvCfg<N, T>::smem) : 0;
                launch_after(pdl, kern, dim3((unsigned)lines, nb), 32, ConvCfg<N, T>::smem, st, ms, want_phys, want_cfl, pf);
                return;
            }
            auto go = [&](auto lpwc) {
                constexpr int LPW = decltype(lpwc)::value;
                const long long nl = (lines + LPW - 1) / LPW;
                // L2 prefetch distance: one wave of resident CTAs (single simulations)
                const long long pf = CAP == 1 ? LPW * resident_ctas(k_xpass<N, T, CAP, false, LPW>, 32, smem_kx<N, T, LPW>()) : 0;
                launch_after(pdl, k_xpass<N, T, CAP, false, LPW>, dim3((unsigned)nl, nb), 32, smem_kx<N, T, LPW>(), st, ms,
                             want_phys, want_cfl, pf, (double*)nullptr);
            };
            if constexpr (xlpw_len<N>()) {
                const int lpw = g.xlpw > 0 ? g.xlpw : XCfg<N, T>::lpw;
                if (lpw == 4) go(std::integral_constant<int, 4>{});
                else if (lpw == 2) go(std::integral_constant<int, 2>{});
                else go(std::integral_constant<int, 1>{});
            } else {
                go(std::integral_constant<int, XCfg<N, T>::lpw>{});
            }
        }
    });
}

// The x pass of the real-space statistics (single simulation): the moments of every
// point into `rs` (kRsSlots x kRsWords doubles, zeroed by the caller).
template <int N, class T> cudaError_t xpass_stats_n(const Geo& g, const Member<T>* M, double* rs, cudaStream_t st) {
    const long long lines = (long long)g.ny * g.nz;
    constexpr size_t sm = sizeof(typename Cplx<T>::type) * 3 * (size_t)xas<N>();
    cudaError_t e = set_smem(k_xpass<N, T, 1, true>, sm);
    if (e) return e;
    MemberSet<T, 1> ms;
    ms.m[0] = M[0];
    k_xpass<N, T, 1, true><<<dim3((unsigned)lines, 1), 32, sm, st>>>(ms, 0, 0, 0, rs);
    return cudaGetLastError();
}

template <int N, class T> cudaError_t ypass_fwd_n(const Geo& g, const Member<T>* M, int B, cudaStream_t st, bool pdl) {
    return for_member_sets(M, B, [&](const auto& ms, int nb) {
        constexpr int CAP = PD_CAP(ms);
        if constexpr (CAP == 1 || batch_len<N>()) {
            const dim3 grid(TCfg<N, 1>::template tiles<T>(g), g.nz, 3 * nb);
            constexpr int NT = TCfg<N, 1>::template nt<T>();
            constexpr size_t sm = TCfg<N, 1>::template smem<T>();
            if constexpr (cube_len<N, T>()) {
                if (is_cube(g, N)) { launch_after(pdl, k_ypass_fwd<N, T, CAP, N>, grid, NT, sm, st, ms); return; }
            }
            launch_after(pdl, k_ypass_fwd<N, T, CAP>, grid, NT, sm, st, ms);
        }
    });
}

// K5a: forward z transforms (mode 1: NL-hat into rk, the transform test hook).
template <int N, class T>
cudaError_t zpass_fwd_n(const Geo& g, const Member<T>* M, int B, int mode, cudaStream_t st, bool pdl) {
    return for_member_sets(M, B, [&](const auto& ms, int nb) {
        constexpr int CAP = PD_CAP(ms);
        if constexpr (CAP == 1 || batch_len<N>())
            launch_after(pdl, k_zpass_fwd<N, T, CAP>, dim3(TCfg<N, 2>::template tiles<T>(g), g.nkj, 3 * nb),
                         TCfg<N, 2>::template nt<T>(), TCfg<N, 2>::template smem<T>(), st, ms, mode);
    });
}
#undef PD_CAP

#define PD_PASSES_INST_T(N, T)                                                                            \
    template cudaError_t configure_n<N, T>(const Geo&);                                                   \
    template cudaError_t zpass_inv_n<N, T>(const Geo&, const Member<T>*, int, int, cudaStream_t, const ZMaps*, bool); \
    template cudaError_t ypass_inv_n<N, T>(const Geo&, const Member<T>*, int, cudaStream_t, bool);              \
    template cudaError_t xpass_n<N, T>(const Geo&, const Member<T>*, int, int, int, cudaStream_t, bool);        \
    template cudaError_t xpass_stats_n<N, T>(const Geo&, const Member<T>*, double*, cudaStream_t);        \
    template cudaError_t ypass_fwd_n<N, T>(const Geo&, const Member<T>*, int, cudaStream_t, bool);              \
    template cudaError_t zpass_fwd_n<N, T>(const Geo&, const Member<T>*, int, int, cudaStream_t, bool);
#define PD_PASSES_INST(N) PD_PASSES_INST_T(N, double) PD_PASSES_INST_T(N, float)

}  // namespace pd
