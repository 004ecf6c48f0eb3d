// api_adjoint.cu -- the misfit-gradient drivers of the C ABI: receiver
// recordings, checkpointed forward runs, segment replays and the reverse
// sweeps of the elastic-wave and heat adjoints (adjoint.cu, heat_adjoint.cu).
#include "api_internal.h"

using namespace b2r_api;

extern "C" {

namespace {


b2r_status adj_check(b2r_handle* h)
{
    if (!h) return fail(nullptr, B2R_ERR_ARG, "null handle");
    if (h->cfg.model != B2R_MODEL_EQWP_STAG)
        return fail(h, B2R_ERR_ARG, "the adjoint covers the staggered elastic-wave model");
    if (h->L.nblk != 1 || h->cfg.R != 1)
        return fail(h, B2R_ERR_ARG, "the adjoint runs on one block with R = 1");
    return B2R_OK;
}

// receiver element offsets (global interior coordinates -> block storage)
b2r_status rec_offsets(b2r_handle* h, int nrec, const int* rec_xyz, std::vector<long long>& idx)
{
    idx.resize(nrec);
    for (int r = 0; r < nrec; ++r) {
        int c[3];
        for (int a = 0; a < 3; ++a) {
            c[a] = rec_xyz[3 * r + a];
            if (c[a] < 0 || c[a] >= h->cfg.env[a]) return fail(h, B2R_ERR_ARG, "receiver %d outside the domain", r);
            c[a] += h->L.H;
        }
        idx[r] = (long long)c[2] * h->L.plane + (long long)c[1] * h->L.P + h->L.xoff + c[0];
    }
    return B2R_OK;
}

}  // namespace

b2r_status b2r_eqwp_record(b2r_handle* h, int nsteps, int nrec, const int* rec_xyz, float* d_out)
{
    b2r_status st;
    if ((st = adj_check(h)) != B2R_OK) return st;
    if (nsteps < 0 || nrec <= 0 || !rec_xyz || !d_out) return fail(h, B2R_ERR_ARG, "invalid receivers");
    std::vector<long long> idx;
    if ((st = rec_offsets(h, nrec, rec_xyz, idx)) != B2R_OK) return st;
    DevBuf d_idx, d_rec;
    CK(h, cudaMalloc(&d_idx.p, sizeof(long long) * nrec));
    CK(h, cudaMalloc(&d_rec.p, sizeof(float) * (size_t)nrec * (nsteps > 0 ? nsteps : 1)));
    CK(h, cudaMemcpyAsync(d_idx.p, idx.data(), sizeof(long long) * nrec, cudaMemcpyHostToDevice, h->stream));
    h->ts = 0;
    for (int n = 0; n < nsteps; ++n) {
        if ((st = substep(h, 0)) != B2R_OK) return st;
        h->ts++;
        CK(h, adjoint_sample(h->fld[B2R_F_VY], (const long long*)d_idx.p, nrec, (float*)d_rec.p + (size_t)n * nrec,
                             h->stream));
    }
    CK(h, cudaMemcpyAsync(d_out, d_rec.p, sizeof(float) * (size_t)nrec * nsteps, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return check_status(h);
}

b2r_status b2r_eqwp_misfit_gradient(b2r_handle* h, int nsteps, int nrec, const int* rec_xyz,
                                    const float* d_obs, int ckpt_every, double* misfit,
                                    double* grad_lambda, double* grad_mu, double* grad_rho,
                                    float* d_syn)
{
    b2r_status st;
    if ((st = adj_check(h)) != B2R_OK) return st;
    if (nsteps <= 0 || nrec <= 0 || !rec_xyz || !d_obs) return fail(h, B2R_ERR_ARG, "invalid receivers / steps");
    const int K = ckpt_every > 0 ? std::min(ckpt_every, nsteps) : nsteps;
    std::vector<long long> idx;
    if ((st = rec_offsets(h, nrec, rec_xyz, idx)) != B2R_OK) return st;
    const size_t fb = field_bytes(h);
    const size_t nseg = (size_t)(nsteps + K - 1) / K;
    // workspace, carved from one allocation kept on the handle: checkpoints
    // (9 fields each), the velocities v^{n0+k} (k = 1..K; k = 0 is the
    // checkpoint) and stencil sums of a segment, the replay's stresses, the
    // adjoint fields, the FP64 gradients as stored and as returned, receivers.
    // Two segment buffers when the workspace fits: segment s-1 is replayed on a
    // second stream while segment s runs its reverse steps.
    const auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t gbytes = (size_t)h->L.bstride * sizeof(double);
    const size_t ncell = (size_t)h->cfg.env[0] * h->cfg.env[1] * h->cfg.env[2];
    const size_t nf_ckpt = nseg * 9, nf_v = (size_t)K * 3, nf_a = (size_t)K * 3;
    const size_t fba = up(fb), gba = up(gbytes);
    const size_t rb = up(sizeof(float) * (size_t)nrec * nsteps), ib = up(sizeof(long long) * nrec);
    int nbuf = nseg > 1 ? 2 : 1;
    for (;; --nbuf) {
        const size_t nfields = nf_ckpt + nbuf * (nf_v + nf_a) + 6 + 18 + 3;
        const size_t need = nfields * fba + 3 * gba + up(ncell * sizeof(double)) + 2 * rb + ib;
        if (h->adj_ws_bytes >= need) break;
        if (h->adj_ws) cudaFree(h->adj_ws);
        h->adj_ws = nullptr;
        h->adj_ws_bytes = 0;
        if (cudaMalloc(&h->adj_ws, need) == cudaSuccess) {
            h->adj_ws_bytes = need;
            break;
        }
        cudaGetLastError();
        h->adj_ws = nullptr;
        if (nbuf == 1) return fail(h, B2R_ERR_OOM, "misfit gradient needs %zu bytes of workspace", need);
    }
    char* ws = static_cast<char*>(h->adj_ws);
    auto take = [&](size_t bytes) {
        char* p = ws;
        ws += bytes;
        return p;
    };
    auto carve = [&](size_t n, std::vector<float*>& out) {
        out.resize(n);
        for (float*& p : out) p = reinterpret_cast<float*>(take(fba));
    };
    std::vector<float*> ckpt, vrep, arep, srep, tmp;
    carve(nf_ckpt, ckpt);
    carve(nf_v * nbuf, vrep);   // buffer b: entries [b * nf_v, (b + 1) * nf_v)
    carve(nf_a * nbuf, arep);
    carve(6, srep);
    carve(18, tmp);
    std::vector<float*> g32;            // FP32 partial gradient sums, folded into gp
    carve(3, g32);
    double* gp[3];
    for (double*& g : gp) g = reinterpret_cast<double*>(take(gba));
    double* const d_out = reinterpret_cast<double*>(take(up(ncell * sizeof(double))));
    float* const d_rec = reinterpret_cast<float*>(take(rb));
    float* const d_res = reinterpret_cast<float*>(take(rb));
    long long* const didx = reinterpret_cast<long long*>(take(ib));
    CK(h, cudaMemsetAsync(tmp[0], 0, 21 * fba + 3 * gba, h->stream));   // tmp, g32 and gp
    // shell cells never change: every velocity of a segment has the initial
    // ones (the sums are read where they are written)
    const long long vstride = (long long)(3 * fba / sizeof(float));
    for (int f = 0; f < 3; ++f)
        CK(h, launch_heat_shell(h->fld[B2R_F_VX + f], vrep[f], vstride, K * nbuf, h->L, h->shell, h->stream));
    CK(h, cudaMemcpyAsync(didx, idx.data(), sizeof(long long) * nrec, cudaMemcpyHostToDevice, h->stream));

    const EqwpStagParams sp = stag_params(h);
    // v^{n0+k} of segment sgi: the checkpoint's velocities for k = 0, slot k of
    // the segment's buffer after
    auto vslot = [&](long long sgi, int k, int f) -> float* {
        return k == 0 ? ckpt[sgi * 9 + B2R_F_VX + f] : vrep[(size_t)(sgi % nbuf) * nf_v + (size_t)(k - 1) * 3 + f];
    };
    auto aslot = [&](long long sgi, int k) -> float* const* {
        return &arep[(size_t)(sgi % nbuf) * nf_a + (size_t)k * 3];
    };
    // every step of a segment with its velocities and stencil sums kept; s6: the
    // checkpoint's stresses, updated in place
    auto replay = [&](long long sgi, float* const* s6, cudaStream_t st) -> b2r_status {
        const int n0 = (int)sgi * K, n1 = std::min(nsteps, n0 + K);
        for (int n = n0; n < n1; ++n) {
            const int k = n - n0;
            const float* vin[3] = {vslot(sgi, k, 0), vslot(sgi, k, 1), vslot(sgi, k, 2)};
            float* vout[3] = {vslot(sgi, k + 1, 0), vslot(sgi, k + 1, 1), vslot(sgi, k + 1, 2)};
            CK(h, launch_eqwp_stag_step_replay(vin, s6, vout, aslot(sgi, k), h->mat, h->L, n, sp, st));
        }
        return B2R_OK;
    };
    auto replay_again = [&](long long sgi, cudaStream_t st) -> b2r_status {
        for (int f = 0; f < 6; ++f)
            CK(h, cudaMemcpyAsync(srep[f], ckpt[sgi * 9 + B2R_F_SXX + f], fb, cudaMemcpyDeviceToDevice, st));
        return replay(sgi, srep.data(), st);
    };

    // forward with checkpoints every K steps and receiver samples; the last
    // nbuf segments are kept as they are stepped, so they need no replay
    const long long slast = (long long)nseg - 1, kept = (long long)nseg - nbuf;
    h->ts = 0;
    for (long long sgi = 0; sgi <= slast; ++sgi) {
        const int n0 = (int)sgi * K, n1 = std::min(nsteps, n0 + K);
        for (int f = 0; f < 9; ++f)
            CK(h, cudaMemcpyAsync(ckpt[sgi * 9 + f], h->fld[f], fb, cudaMemcpyDeviceToDevice, h->stream));
        for (int n = n0; n < n1 && sgi < kept; ++n) {
            if ((st = substep(h, 0)) != B2R_OK) return st;
            h->ts++;
            CK(h, adjoint_sample(h->fld[B2R_F_VY], didx, nrec, d_rec + (size_t)n * nrec, h->stream));
        }
        if (sgi < kept) continue;
        if ((st = replay(sgi, h->fld + B2R_F_SXX, h->stream)) != B2R_OK) return st;
        CK(h, adjoint_sample(vslot(sgi, 1, 1), didx, nrec, d_rec + (size_t)n0 * nrec, h->stream, n1 - n0, vstride));
        for (int f = 0; f < 3; ++f)
            CK(h, cudaMemcpyAsync(h->fld[B2R_F_VX + f], vslot(sgi, n1 - n0, f), fb, cudaMemcpyDeviceToDevice,
                                  h->stream));
    }

    // reverse sweep, segment by segment, those not kept replayed forward from
    // their checkpoint into segment buffer sgi % nbuf first.  With two buffers
    // the replay of the segment below runs on a second stream while this
    // segment's reverse steps run; the results are the same bits.
    struct AuxStream {
        cudaStream_t s = nullptr;
        cudaEvent_t rep[2] = {}, rev[2] = {};
        ~AuxStream()
        {
            for (cudaEvent_t e : {rep[0], rep[1], rev[0], rev[1]})
                if (e) cudaEventDestroy(e);
            if (s) cudaStreamDestroy(s);
        }
    } ax;
    if (nbuf == 2) {
        CK(h, cudaStreamCreateWithFlags(&ax.s, cudaStreamNonBlocking));
        for (cudaEvent_t* e : {&ax.rep[0], &ax.rep[1], &ax.rev[0], &ax.rev[1]})
            CK(h, cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    }
    // misfit and residual (host, FP64)
    std::vector<float> syn((size_t)nrec * nsteps), res((size_t)nrec * nsteps);
    CK(h, cudaMemcpyAsync(syn.data(), d_rec, sizeof(float) * syn.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    double J = 0.0;
    for (size_t i = 0; i < syn.size(); ++i) {
        const double r = (double)syn[i] - (double)d_obs[i];
        res[i] = (float)r;
        J += 0.5 * r * r;
    }
    if (misfit) *misfit = J;
    if (d_syn) std::copy(syn.begin(), syn.end(), d_syn);
    CK(h, cudaMemcpyAsync(d_res, res.data(), sizeof(float) * res.size(), cudaMemcpyHostToDevice, h->stream));

    float* const* tp = tmp.data();
    const float* mat[3] = {h->mat[0], h->mat[1], h->mat[2]};
    const float dt_h = (float)(h->cfg.dt / h->cfg.h);
    CK(h, adjoint_inject(tp[1], didx, nrec, d_res + (size_t)(nsteps - 1) * nrec, h->stream));
    for (long long sgi = slast; sgi >= 0; --sgi) {
        const int n0 = (int)sgi * K;
        const int n1 = std::min(nsteps, n0 + K);
        if (nbuf == 1 && sgi < kept && (st = replay_again(sgi, h->stream)) != B2R_OK) return st;
        if (nbuf == 2 && sgi < kept) CK(h, cudaStreamWaitEvent(h->stream, ax.rep[sgi % 2], 0));
        if (nbuf == 2 && sgi >= 1 && sgi <= kept) {
            const int b1 = (int)((sgi - 1) % 2);
            // that buffer last served segment sgi + 1, whose reverse steps are queued
            CK(h, cudaStreamWaitEvent(ax.s, ax.rev[b1], 0));
            if ((st = replay_again(sgi - 1, ax.s)) != B2R_OK) return st;
            CK(h, cudaEventRecord(ax.rep[b1], ax.s));
        }
        for (int n = n1 - 1; n >= n0; --n) {
            const int k = n - n0;
            const float* vn[3] = {vslot(sgi, k, 0), vslot(sgi, k, 1), vslot(sgi, k, 2)};
            float* const* a = aslot(sgi, k);
            const float* an[3] = {a[0], a[1], a[2]};
            CK(h, adjoint_step(tp, vn, an, mat, g32.data(), h->L, dt_h, n == 0, h->adj_fused, didx, nrec,
                               n > 0 ? d_res + (size_t)(n - 1) * nrec : nullptr, h->stream));
            // the partial sums into FP64 on a fixed schedule of step numbers
            // (step 0 is the last reverse step, so nothing is left behind)
            if (n % adjoint_fold_steps() == 0) CK(h, adjoint_fold(g32.data(), gp, h->L, h->stream));
        }
        if (nbuf == 2) CK(h, cudaEventRecord(ax.rev[sgi % 2], h->stream));
    }
    // gradients out (interior cells, x fastest), g_rho = -g_b / rho^2
    double* outs[3] = {grad_lambda, grad_mu, grad_rho};
    for (int m = 0; m < 3; ++m) {
        if (!outs[m]) continue;
        CK(h, adjoint_grad_out(gp[m], h->mat[2], m == 2, h->L, d_out, h->stream));
        CK(h, cudaMemcpyAsync(outs[m], d_out, ncell * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    }
    CK(h, cudaStreamSynchronize(h->stream));
    h->ts = nsteps;
    h->halos_fresh = false;
    h->upmask = 0;
    return check_status(h);
}

namespace {

b2r_status heat_adj_check(b2r_handle* h)
{
    if (!h) return fail(nullptr, B2R_ERR_ARG, "null handle");
    if (h->cfg.model != B2R_MODEL_HEAT) return fail(h, B2R_ERR_ARG, "the heat adjoint needs the heat model");
    if (h->L.nblk != 1 || h->L.periodic)
        return fail(h, B2R_ERR_ARG, "the heat adjoint runs on one block with a fixed shell");
    return ensure_kappa(h);
}

HeatLap heat_lap_of(const b2r_handle* h)
{
    return heat_lap(h->cfg.D, h->cfg.alpha_dt, h->cfg.dx, h->cfg.dy, h->cfg.dz);
}

}  // namespace

b2r_status b2r_heat_record(b2r_handle* h, int nsteps, int nrec, const int* rec_xyz, float* d_out)
{
    b2r_status st;
    if ((st = heat_adj_check(h)) != B2R_OK) return st;
    if (nsteps < 0 || nrec <= 0 || !rec_xyz || !d_out) return fail(h, B2R_ERR_ARG, "invalid receivers");
    std::vector<long long> idx;
    if ((st = rec_offsets(h, nrec, rec_xyz, idx)) != B2R_OK) return st;
    DevBuf d_idx, d_rec;
    CK(h, cudaMalloc(&d_idx.p, sizeof(long long) * nrec));
    CK(h, cudaMalloc(&d_rec.p, sizeof(float) * (size_t)nrec * (nsteps > 0 ? nsteps : 1)));
    CK(h, cudaMemcpyAsync(d_idx.p, idx.data(), sizeof(long long) * nrec, cudaMemcpyHostToDevice, h->stream));
    const HeatLap c = heat_lap_of(h);
    const long long* didx = (const long long*)d_idx.p;
    float* rec = (float*)d_rec.p;
    for (int n = 0; n < nsteps; ++n) {   // a step samples the receivers of the one before
        CK(h, launch_heat_kappa_step(static_cast<float*>(h->buf[h->cur]), static_cast<float*>(h->buf[1 - h->cur]),
                                     h->mat[0], h->L, h->cfg.D, c, didx, nrec,
                                     n > 0 ? rec + (size_t)(n - 1) * nrec : nullptr, h->stream));
        h->cur = 1 - h->cur;
    }
    if (nsteps > 0)
        CK(h, adjoint_sample(static_cast<float*>(h->buf[h->cur]), didx, nrec, rec + (size_t)(nsteps - 1) * nrec,
                             h->stream));
    h->ts += nsteps;
    CK(h, cudaMemcpyAsync(d_out, d_rec.p, sizeof(float) * (size_t)nrec * nsteps, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return check_status(h);
}

b2r_status b2r_heat_misfit_gradient(b2r_handle* h, int nsteps, int nrec, const int* rec_xyz,
                                    const float* d_obs, int ckpt_every, double* misfit,
                                    double* grad_kappa, float* d_syn)
{
    b2r_status st;
    if ((st = heat_adj_check(h)) != B2R_OK) return st;
    if (nsteps <= 0 || nrec <= 0 || !rec_xyz || !d_obs) return fail(h, B2R_ERR_ARG, "invalid receivers / steps");
    const int K = ckpt_every > 0 ? std::min(ckpt_every, nsteps) : nsteps;
    std::vector<long long> idx;
    if ((st = rec_offsets(h, nrec, rec_xyz, idx)) != B2R_OK) return st;
    const size_t fb = field_bytes(h);
    const size_t nseg = (size_t)(nsteps + K - 1) / K;
    // workspace on the handle: checkpoints 1 .. nseg-1 (checkpoint 0 is the
    // caller's field, which no step overwrites), segment states 1 .. K, lam,
    // two y buffers, the FP64 gradient as stored and as returned, receivers
    const auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t fba = up(fb), gb = (size_t)h->L.bstride * sizeof(double);
    const size_t ncell = (size_t)h->cfg.env[0] * h->cfg.env[1] * h->cfg.env[2];
    const size_t nstate = (nseg - 1) + (size_t)K;
    const size_t rb = up(sizeof(float) * (size_t)nrec * nsteps), ib = up(sizeof(long long) * nrec);
    const size_t need = (nstate + 3) * fba + up(gb) + up(ncell * sizeof(double)) + 2 * rb + ib;
    if (h->adj_ws_bytes < need) {
        if (h->adj_ws) cudaFree(h->adj_ws);
        h->adj_ws = nullptr;
        h->adj_ws_bytes = 0;
        if (cudaMalloc(&h->adj_ws, need) != cudaSuccess) {
            cudaGetLastError();
            return fail(h, B2R_ERR_OOM, "heat gradient needs %zu bytes of workspace", need);
        }
        h->adj_ws_bytes = need;
    }
    char* ws = static_cast<char*>(h->adj_ws);
    auto carve = [&](size_t bytes) {
        char* p = ws;
        ws += bytes;
        return p;
    };
    float* const u0 = static_cast<float*>(h->buf[h->cur]);
    float* const states = reinterpret_cast<float*>(carve(nstate * fba));
    const long long fstride = (long long)(fba / sizeof(float));
    auto ckpt = [&](long long sgi) { return sgi == 0 ? u0 : states + (sgi - 1) * fstride; };
    auto slot = [&](int k) { return states + ((long long)nseg - 1 + k - 1) * fstride; };   // k = 1 .. K
    float* const lam = reinterpret_cast<float*>(carve(fba));
    float* yb[2];
    for (float*& b : yb) b = reinterpret_cast<float*>(carve(fba));
    double* const g = reinterpret_cast<double*>(carve(up(gb)));
    double* const d_out = reinterpret_cast<double*>(carve(up(ncell * sizeof(double))));
    float* const d_rec = reinterpret_cast<float*>(carve(rb));
    float* const d_res = reinterpret_cast<float*>(carve(rb));
    long long* const didx = reinterpret_cast<long long*>(carve(ib));
    CK(h, cudaMemsetAsync(lam, 0, 3 * fba, h->stream));   // and both y
    CK(h, cudaMemsetAsync(g, 0, gb, h->stream));
    CK(h, cudaMemcpyAsync(didx, idx.data(), sizeof(long long) * nrec, cudaMemcpyHostToDevice, h->stream));
    const HeatLap c = heat_lap_of(h);
    const int D = h->cfg.D;
    // shell cells never change: every state has the initial one's
    CK(h, launch_heat_shell(u0, states, fstride, (int)nstate, h->L, D, h->stream));

    // forward: state n is a checkpoint at multiples of K, its segment's slot
    // in the last segment (which needs no replay), and one of two slots in
    // turn otherwise; a step samples the receivers of the one before
    const int n_last = (int)(nseg - 1) * K;
    auto state = [&](int n) {
        if (n % K == 0 && n < nsteps) return ckpt(n / K);
        return slot(n > n_last ? n - n_last : 1 + n % 2);
    };
    for (int n = 0; n < nsteps; ++n)
        CK(h, launch_heat_kappa_step(state(n), state(n + 1), h->mat[0], h->L, D, c, didx, nrec,
                                     n > 0 ? d_rec + (size_t)(n - 1) * nrec : nullptr, h->stream));
    CK(h, adjoint_sample(state(nsteps), didx, nrec, d_rec + (size_t)(nsteps - 1) * nrec, h->stream));
    std::vector<float> syn((size_t)nrec * nsteps), res((size_t)nrec * nsteps);
    CK(h, cudaMemcpyAsync(syn.data(), d_rec, sizeof(float) * syn.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    double J = 0.0;
    for (size_t i = 0; i < syn.size(); ++i) {
        const double r = (double)syn[i] - (double)d_obs[i];
        res[i] = (float)r;
        J += 0.5 * r * r;
    }
    if (misfit) *misfit = J;
    if (d_syn) std::copy(syn.begin(), syn.end(), d_syn);
    CK(h, cudaMemcpyAsync(d_res, res.data(), sizeof(float) * res.size(), cudaMemcpyHostToDevice, h->stream));

    // reverse sweep, segment by segment, each but the last replayed first
    int cur = 0;   // y buffer of the step
    for (long long sgi = (long long)nseg - 1; sgi >= 0; --sgi) {
        const int n0 = (int)sgi * K;
        const int n1 = std::min(nsteps, n0 + K);
        auto u_at = [&](int k) { return k == 0 ? ckpt(sgi) : slot(k); };
        if (sgi < (long long)nseg - 1)
            for (int n = n0; n + 1 < n1; ++n)
                CK(h, launch_heat_kappa_step(u_at(n - n0), u_at(n - n0 + 1), h->mat[0], h->L, D, c, didx, 0, nullptr,
                                             h->stream));
        for (int n = n1 - 1; n >= n0; --n) {
            CK(h, launch_heat_adjoint_inject(lam, yb[cur], h->mat[0], didx, nrec, d_res + (size_t)n * nrec, h->stream));
            CK(h, launch_heat_adjoint_step(lam, yb[cur], yb[1 - cur], u_at(n - n0), h->mat[0], g, h->L, D, c, h->stream));
            cur = 1 - cur;
        }
    }
    if (grad_kappa) {
        CK(h, adjoint_grad_out(g, nullptr, 0, h->L, d_out, h->stream));
        CK(h, cudaMemcpyAsync(grad_kappa, d_out, ncell * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    }
    CK(h, cudaStreamSynchronize(h->stream));
    h->ts = nsteps;
    return check_status(h);
}

}  // extern "C"
