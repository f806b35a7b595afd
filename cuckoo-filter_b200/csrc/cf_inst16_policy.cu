// cf_inst16_policy.cu -- kernels for 16-bit tags under the AddSub and Offset policies (bucket_policy_benchmark.cu:16-17) (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits16_policy(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 16, 16, 8, ALT_ADDSUB>>::table());
    v.push_back(Launchers<Cfg<4, 16, 16, 8, ALT_ADDSUB>>::table());
    v.push_back(Launchers<Cfg<8, 16, 16, 8, ALT_OFFSET>>::table());
    v.push_back(Launchers<Cfg<4, 16, 16, 8, ALT_OFFSET>>::table());
}

}  // namespace cfb
