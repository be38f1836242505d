// functor_plugin.cu -- force plugins whose pair functor is built on one of the
// library's, for the tests:
//   variant 0  a functor that derives from psim::LJPair and gives its own
//              fnet64 and fnet32: the Yukawa term alone
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

class Functor : public psim::PluginForce<Functor, TailPair> {
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
        TailPair t;
        static_cast<psim::LJPair&>(t) = psim::make_lj_pair(
            p.kT, p.well_depth, p.lj_num, p.yukawa_strength, p.debye_length, p.cutoff);
        return f(t);
    }
};

}  // namespace

PSIM_FORCE_PLUGIN(Functor)
