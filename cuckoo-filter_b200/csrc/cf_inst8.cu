// cf_inst8.cu -- kernels for 8-bit tags in buckets of 8 and 16 slots (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits8(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 8, 8, 8>>::table());
    v.push_back(Launchers<Cfg<4, 8, 8, 8>>::table());
    v.push_back(Launchers<Cfg<8, 8, 16, 8>>::table());
    v.push_back(Launchers<Cfg<4, 8, 16, 8>>::table());
}

}  // namespace cfb
