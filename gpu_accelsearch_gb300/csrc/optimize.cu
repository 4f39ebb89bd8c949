// optimize.cu -- host side of candidate refinement and properties
// (accel_optimize_candidates; the kernels are in refine.cu).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "../../include/accelsearch.h"
#include "context.h"

extern "C" int accel_trial_spectrum(accel_ctx* c, int trial, const accel_complex** spec, long long* numbins) {
    if (!c || !spec || !numbins) return set_error(ACCEL_ERR_INVALID, "accel_trial_spectrum: null argument");
    if (trial < 0 || trial >= c->last_trials || trial >= (int)c->trials.size())
        return set_error(ACCEL_ERR_INVALID, "accel_trial_spectrum: trial %d not in the last search", trial);
    *spec = reinterpret_cast<const accel_complex*>(c->trials[trial].spec);
    *numbins = c->trials[trial].numbins;
    return ACCEL_OK;
}

extern "C" int accel_optimize_candidates(accel_ctx* c, int ntrials, const accel_complex* const* wspec,
                                         const long long* numbins, const long long* rlo, const double* tobs,
                                         const accel_candidate* in, long long n, int refine,
                                         accel_optimized* out) {
    if (!c || ntrials < 1 || !wspec || !numbins || !rlo || !tobs || n < 0 || (n > 0 && (!in || !out)))
        return set_error(ACCEL_ERR_INVALID, "accel_optimize_candidates: bad argument");
    if (n > 0x7fffffffLL) return set_error(ACCEL_ERR_INVALID, "accel_optimize_candidates: too many candidates");
    for (int t = 0; t < ntrials; t++)
        if (!wspec[t] || numbins[t] < 1 || !(tobs[t] > 0.0))
            return set_error(ACCEL_ERR_INVALID, "accel_optimize_candidates: trial %d", t);
    int rc = ensure_device(c);
    if (rc) return rc;
    std::vector<OptCand> cand((size_t)n);
    const double zreach = refine ? 2.63 : 0.0;  // how far the grids reach in z
    int maxharm = 1, maxdata = 1;
    // the candidates in launch order: those whose windows suit the node rule,
    // then the wider ones, for the direct form.  Each goes by its own width,
    // so that what else is in the list changes neither its result nor its cost.
    // (empty without wide ones: as given)
    std::vector<long long> order, wide;
    for (long long i = 0; i < n; i++) {
        const accel_candidate& x = in[i];
        if (x.trial < 0 || x.trial >= ntrials || x.numharm < 1 || x.numharm > c->nh ||
            (x.numharm & (x.numharm - 1)) || x.step < 0 || !std::isfinite(x.r) || !std::isfinite(x.z))
            return set_error(ACCEL_ERR_INVALID, "accel_optimize_candidates: candidate %lld", i);
        OptCand& o = cand[i];
        o.r = x.r;
        o.z = x.z;
        o.numharm = x.numharm;
        o.trial = x.trial;
        maxharm = std::max(maxharm, x.numharm);
        int maxpanels = 0;
        // harmonic k of H is the bank's harmonic p/q = k/H in lowest terms;
        // its segment in the candidate's step is the search's (A6/A7)
        const long long startr = rlo[x.trial] + (long long)x.step * (c->uselen / 2);
        for (int k = 1; k <= x.numharm; k++) {
            const int g = std::gcd(k, x.numharm), p = k / g, q = x.numharm / g;
            int h = 0;
            while (h < c->nh && !(c->hp[h].p == p && c->hp[h].q == q)) h++;
            if (h == c->nh) return set_error(ACCEL_ERR_INVALID, "accel_optimize_candidates: harmonic %d/%d", p, q);
            const StepHarm sh = step_harm(startr, c->uselen, p, q, c->hp[h].hw0);
            o.lobin[k - 1] = sh.lobin;
            o.numdata[k - 1] = std::min(sh.numdata, c->hp[h].M);
            maxdata = std::max(maxdata, o.numdata[k - 1]);
            o.panels[k - 1] = refine_panels(x.z * k / x.numharm, zreach * k / x.numharm);
            maxpanels = std::max(maxpanels, o.panels[k - 1]);
        }
        if (maxpanels > (refine ? kRefineMaxPanels : kRefineMaxPanelsPoint)) wide.push_back(i);
    }
    if (n == 0) return ACCEL_OK;
    const long long nnear = n - (long long)wide.size();
    if (!wide.empty()) {
        for (long long i = 0, w = 0; i < n; i++) {
            if (w < (long long)wide.size() && wide[w] == i) w++;
            else order.push_back(i);
        }
        order.insert(order.end(), wide.begin(), wide.end());
    }
    auto at = [&](long long j) { return order.empty() ? j : order[j]; };
    // launches of at most kOptBatch candidates and kOptNodes nodes, from one
    // workspace kept by the context: spectra table, candidates, results,
    // norms and node values (256 MB of those; with 64 MB a list of 1000
    // candidates took 7.6 ms instead of 7.4: more launches end in a part wave)
    constexpr long long kOptBatch = 1 << 16, kOptNodes = 1LL << 21;
    long long most = 0, most_nodes = 0;
    std::vector<long long> ends;  // end of each launch's candidates
    for (long long i = 0; i < n;) {
        const bool direct = i >= nnear;
        const long long end = std::min(direct ? n : nnear, i + kOptBatch);
        long long nodes = 0, j = i;
        for (; j < end; j++) {
            OptCand& o = cand[at(j)];
            long long own = 0;
            for (int k = 0; k < o.numharm && !direct; k++) own += (long long)o.panels[k] * kRefineNodes;
            if (j > i && nodes + own > kOptNodes) break;
            o.scratch_off = nodes;
            nodes += own;
        }
        most = std::max(most, j - i);
        most_nodes = std::max(most_nodes, nodes);
        ends.push_back(j);
        i = j;
    }
    auto pad = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t off_nb = pad(sizeof(float2*) * ntrials), off_in = off_nb + pad(sizeof(long long) * ntrials),
                 off_out = off_in + pad(sizeof(OptCand) * most), off_norm = off_out + pad(sizeof(OptOut) * most),
                 off_s = off_norm + pad(sizeof(double) * kMaxHarm * most),
                 dev_bytes = off_s + sizeof(double2) * kRefineValues * most_nodes, host_bytes = off_norm;
    cudaError_t e = cudaSuccess;
    if (dev_bytes > c->opt_dev_cap) {
        cudaFree(c->opt_dev);
        c->opt_dev = nullptr;
        c->opt_dev_cap = 0;
        e = ctx_malloc(c, &c->opt_dev, dev_bytes);
        if (e == cudaSuccess) c->opt_dev_cap = dev_bytes;
    }
    if (e == cudaSuccess && host_bytes > c->opt_host_cap) {
        cudaFreeHost(c->opt_host);
        c->opt_host = nullptr;
        c->opt_host_cap = 0;
        e = cudaMallocHost(&c->opt_host, host_bytes);
        if (e == cudaSuccess) c->opt_host_cap = host_bytes;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(ACCEL_ERR_NOMEM, "accel_optimize_candidates: %s", cudaGetErrorString(e));
    }
    char* dev = static_cast<char*>(c->opt_dev);
    char* host = static_cast<char*>(c->opt_host);
    std::vector<OptOut> res((size_t)n);
    long long i0 = 0;
    for (long long i1 : ends) {
        const long long m = i1 - i0;
        std::memcpy(host, wspec, sizeof(float2*) * ntrials);
        std::memcpy(host + off_nb, numbins, sizeof(long long) * ntrials);
        OptCand* hin = reinterpret_cast<OptCand*>(host + off_in);
        for (long long j = i0; j < i1; j++) hin[j - i0] = cand[at(j)];
        e = cudaMemcpyAsync(dev, host, off_in + sizeof(OptCand) * m, cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) {
            RefineArgs a{};
            a.spec = reinterpret_cast<const float2* const*>(dev);
            a.numbins = reinterpret_cast<const long long*>(dev + off_nb);
            a.in = reinterpret_cast<const OptCand*>(dev + off_in);
            a.out = reinterpret_cast<OptOut*>(dev + off_out);
            a.norm2 = reinterpret_cast<double*>(dev + off_norm);
            a.scratch = reinterpret_cast<double2*>(dev + off_s);
            a.n = (int)m;
            a.maxharm = maxharm;
            a.refine = refine != 0;
            a.exact_rsqrt = c->cfg.exact_rsqrt;
            a.maxdata = maxdata;
            if ((i0 >= nnear ? launch_refine_direct(a, c->stream) : launch_refine(a, c->stream)) != 0) {
                e = cudaGetLastError();
                if (e == cudaSuccess) e = cudaErrorUnknown;
            }
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host + off_out, dev + off_out, sizeof(OptOut) * m, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess)
            return set_error(ACCEL_ERR_CUDA, "accel_optimize_candidates: %s", cudaGetErrorString(e));
        const OptOut* hout = reinterpret_cast<const OptOut*>(host + off_out);
        for (long long j = i0; j < i1; j++) res[at(j)] = hout[j - i0];
        i0 = i1;
    }
    for (long long i = 0; i < n; i++) {
        const OptOut& o = res[i];
        accel_optimized& y = out[i];
        y.cand = in[i];
        y.cand.r = o.r;
        y.cand.z = o.z;
        y.cand.power = (float)o.power;
        y.cand.sigma = (float)sigma_of_power_host(o.power, in[i].numharm, c->cfg.numindep);
        y.r_grid = in[i].r;
        y.z_grid = in[i].z;
        for (int k = 0; k < 16; k++) y.harm_power[k] = k < kMaxHarm ? o.harm[k] : 0.f;
        const double T = tobs[in[i].trial];
        y.f = o.r / T;
        y.fdot = o.z / (T * T);
        y.period = y.f != 0.0 ? 1.0 / y.f : 0.0;
        y.pdot = y.f != 0.0 ? -y.fdot / (y.f * y.f) : 0.0;
    }
    return ACCEL_OK;
}
