// functor_plugin.cu -- force plugins whose pair functor is built on one of the
// library's, for the tests:
//   variant 0  a functor that derives from psim::LJPair and gives its own
//              fnet64 and fnet32: the Yukawa term alone
//   variant 1  a psim::LJPair whose members the plugin fills itself
//   variant 2  a psim::LJPair made without a Yukawa term and given one afterwards
// The settings are the LennardJones plugin's, and `variant`.
#include "psim_plugin.cuh"

namespace {

struct TailPair : psim::LJPair {
    __host__ __device__ double fnet64(double, double r, double rinv, double) const {
        return -kTwd * (exp(-(r * inv_lambda)) * (rinv * rinv * (lambda + r) * yuk));
    }
    __device__ float fnet32(float, float r, float rinv, float) const {
        return -kTwdf * (__expf(-r * inv_lambdaf) * (rinv * rinv * (lambdaf + r) * yukf));
    }
};

psim::LJPair filled(const psim_force_params& p) {
    psim::LJPair q{};
    q.rc2 = p.cutoff * p.cutoff;
    q.kTwd = p.kT * p.well_depth;
    q.four_n = 4.0 * p.lj_num;
    q.n = p.lj_num;
    q.yuk = p.yukawa_strength;
    q.lambda = p.debye_length;
    q.inv_lambda = 1.0 / p.debye_length;
    q.rc2f = (float)q.rc2;
    q.kTwdf = (float)q.kTwd;
    q.four_nf = (float)q.four_n;
    q.yukf = (float)q.yuk;
    q.lambdaf = (float)q.lambda;
    q.inv_lambdaf = (float)q.inv_lambda;
    return q;
}

class Functor : public psim::PluginForce<Functor, psim::LJPair> {
public:
    explicit Functor(PSim::config* cfg) {
        name = "Functor";
        params_.kind = PSIM_FORCE_PLUGIN;
        params_.kT = cfg->getParam<double>("kT", 1.0);
        params_.well_depth = cfg->getParam<double>("wellDepth", 1.0);
        params_.yukawa_strength = cfg->getParam<double>("yukawaStrength", 3.0);
        params_.lj_num = cfg->getParam<int>("ljNum", 6);
        params_.cutoff = cfg->getParam<double>("cutOff", 2.5);
        params_.debye_length = cfg->getParam<double>("debyeLength", 0.5);
        params_.user[0] = cfg->getParam<int>("variant", 0);
    }
    template <class F>
    static int dispatch(const psim_force_params& p, F&& f) {
        if (p.user[0] == 1) return f(filled(p));
        if (p.user[0] == 2) {
            psim::LJPair q = psim::make_lj_pair(p.kT, p.well_depth, p.lj_num, 0.0,
                                                p.debye_length, p.cutoff);
            q.yuk = p.yukawa_strength;
            q.yukf = (float)q.yuk;
            return f(q);
        }
        TailPair t;
        static_cast<psim::LJPair&>(t) = psim::make_lj_pair(
            p.kT, p.well_depth, p.lj_num, p.yukawa_strength, p.debye_length, p.cutoff);
        return f(t);
    }
};

}  // namespace

PSIM_FORCE_PLUGIN(Functor)
