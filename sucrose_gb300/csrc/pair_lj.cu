// Point-particle pair potentials: lj_, lj12_, ljw_ and wca_
// (fortran/force.f90:6-190), FP32 per pair, FP64 energy sums.
#include <cmath>

#include "pair_point.cuh"

PotLJ<-1> make_pot_lj(const sg_ctx* ctx, const sg_pair_params* p) {
    PotLJ<-1> pot;
    pot.prefiltered = 0;
    pot.pos = ctx->pos;
    pot.b = make_boxf(ctx);
    pot.kind = p->kind;
    pot.sigma = (float)p->sigma;
    pot.eps = (float)p->epsilon;
    pot.rc = (float)p->cutoff;
    pot.rc2 = (float)(p->cutoff * p->cutoff);
    pot.wf = (float)p->wf;
    pot.sig2 = (float)(p->sigma * p->sigma);
    double s = p->sigma, e = p->epsilon, rc = p->cutoff;
    double cut = 0.0;
    if (p->kind == SG_LJ) {
        double c2 = (s * s) / (rc * rc), c6 = c2 * c2 * c2;
        cut = 4.0 * e * (c6 * c6 - c6);
    } else if (p->kind == SG_LJ12) {
        double c2 = (s * s) / (rc * rc), c6 = c2 * c2 * c2;
        cut = e * (c6 * c6 - 2.0 * c6);
    } else if (p->kind == SG_LJW) {
        double c = s / rc, c2 = c * c, c6 = c2 * c2 * c2;
        cut = e * (c6 * c6 - 2.0 * c6);
    }
    pot.pot_cut = (float)cut;
    return pot;
}

int sg_launch_pair_simple(sg_ctx* ctx, const sg_pair_params* p) {
    const PotLJ<-1> pot = make_pot_lj(ctx, p);
    if (ctx->nrep) {
        const PairTune tune = sg_pair_tune_for(ctx, p->kind, true);
        if (!tune.filter) return p->kind == SG_LJ ? launch_spans(ctx, pot_as<PotLJ<SG_LJ>>(pot), tune.block)
                                                  : launch_spans(ctx, pot, tune.block);
    }
    if (!rows_apply(ctx)) return launch_pair(ctx, pot, p->kind);
    if (p->kind == SG_LJ) return launch_rows(ctx, pot_as<PotLJ<SG_LJ>>(pot), p->kind);
    if (p->kind == SG_WCA) return launch_rows(ctx, pot_as<PotLJ<SG_WCA>>(pot), p->kind);
    return launch_rows(ctx, pot, p->kind);
}

// Whether two pair sets run as one pass of the row driver: a set of the
// Lennard-Jones family and one of the charged (or Morse) kinds, on a single
// system with rows. Each neighbour's position is fetched once for both: WCA and
// Coulomb on 131 072 charged spheres 65 us together, 46 and 63 us apart.
bool sg_pair_sets_fuse(const sg_ctx* ctx, const sg_pair_params* a, const sg_pair_params* b) {
    return rows_apply(ctx) && a->kind >= SG_LJ && a->kind <= SG_WCA && b->kind >= SG_MORSE && b->kind <= SG_COULOMB;
}

int sg_launch_pair_both(sg_ctx* ctx, const sg_pair_params* a, const sg_pair_params* b) {
    PotElec<-1> elec;
    const PotLJ<-1> lj = make_pot_lj(ctx, a);
    if (int rc = make_pot_elec(ctx, b, elec)) return rc;
    if (a->kind == SG_WCA && b->kind == SG_COULOMB) {
        PotBoth<PotLJ<SG_WCA>, PotElec<SG_COULOMB>> pot;
        pot.a = pot_as<PotLJ<SG_WCA>>(lj);
        pot.b = pot_as<PotElec<SG_COULOMB>>(elec);
        return launch_rows(ctx, pot, b->kind);
    }
    PotBoth<PotLJ<-1>, PotElec<-1>> pot;
    pot.a = lj;
    pot.b = elec;
    return launch_rows(ctx, pot, b->kind);
}
