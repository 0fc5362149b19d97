// check_devices.cpp -- a per-device record keeps its address and contents while
// records of other devices are made (mrg8g_devices.h).
#include <cstdio>
#include <vector>

#include "mrg8g_devices.h"

struct Record {
    bool ready = false;
    int sms = 0;
    int pad[30] = {};
};

int main() {
    mrg8g::PerDevice<Record> devices;
    std::vector<Record*> kept;
    int bad = 0;
    const int order[] = {0, 2, 1, 7, 63, 8, 64, 500};
    for (int dev : order) {
        Record* r = &devices.at(dev);
        bad += r->ready;  // made empty
        r->ready = true;
        r->sms = 100 + dev;
        kept.push_back(r);
        for (size_t i = 0; i < kept.size(); ++i)
            bad += &devices.at(order[i]) != kept[i] || kept[i]->sms != 100 + order[i];
    }
    std::printf("bad=%d\n", bad);
    return bad != 0;
}
