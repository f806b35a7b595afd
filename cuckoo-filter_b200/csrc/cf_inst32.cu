// cf_inst32.cu -- kernels for 32-bit tags in buckets of 2, 4 and 8 slots (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits32(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 32, 2, 8>>::table());
    v.push_back(Launchers<Cfg<4, 32, 2, 8>>::table());
    v.push_back(Launchers<Cfg<8, 32, 4, 8>>::table());
    v.push_back(Launchers<Cfg<4, 32, 4, 8>>::table());
    v.push_back(Launchers<Cfg<8, 32, 8, 8>>::table());
    v.push_back(Launchers<Cfg<4, 32, 8, 8>>::table());
}

}  // namespace cfb
