// cf_inst16_more.cu -- kernels for 16-bit tags in 64- to 256-byte buckets, and with WordType uint32_t (see cf_registry.cuh).
#include "cf_registry.cuh"

namespace cfb {

void register_bits16_more(std::vector<OpsTable>& v) {
    v.push_back(Launchers<Cfg<8, 16, 32, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 32, 8>>::table());
    v.push_back(Launchers<Cfg<8, 16, 64, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 64, 8>>::table());
    v.push_back(Launchers<Cfg<8, 16, 128, 8>>::table());
    v.push_back(Launchers<Cfg<4, 16, 128, 8>>::table());
    v.push_back(Launchers<Cfg<8, 16, 16, 4>>::table());
    v.push_back(Launchers<Cfg<4, 16, 16, 4>>::table());
}

}  // namespace cfb
