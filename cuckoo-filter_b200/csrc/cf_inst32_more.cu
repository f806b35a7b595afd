// cf_inst32_more.cu -- kernels for 32-bit tags in 16-slot buckets, and with WordType uint32_t (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits32_more(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 32, 16, 8>>::table());
    v.push_back(Launchers<Cfg<4, 32, 16, 8>>::table());
    v.push_back(Launchers<Cfg<8, 32, 8, 4>>::table());
    v.push_back(Launchers<Cfg<4, 32, 8, 4>>::table());
}

}  // namespace cfb
