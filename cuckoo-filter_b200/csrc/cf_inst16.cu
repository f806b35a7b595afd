// cf_inst16.cu -- kernels for 16-bit tags in buckets of 4, 8 and 16 slots (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits16(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 16, 4, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 4, 8>>::table());
    v.push_back(Launchers<Cfg<8, 16, 8, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 8, 8>>::table());
    v.push_back(Launchers<Cfg<8, 16, 16, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 16, 8>>::table());
}

}  // namespace cfb
