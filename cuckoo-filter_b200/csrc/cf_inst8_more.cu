// cf_inst8_more.cu -- kernels for 8-bit tags in wider buckets, and with WordType uint32_t (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits8_more(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 8, 32, 8>>::table());
    v.push_back(Launchers<Cfg<4, 8, 32, 8>>::table());
    v.push_back(Launchers<Cfg<8, 8, 64, 8>>::table());
    v.push_back(Launchers<Cfg<4, 8, 64, 8>>::table());
    v.push_back(Launchers<Cfg<8, 8, 16, 4>>::table());
    v.push_back(Launchers<Cfg<4, 8, 16, 4>>::table());
}

}  // namespace cfb
